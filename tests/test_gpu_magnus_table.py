"""GPU checks of Magnus-4 against the oracle at the edges of its paths: the staged sums and
differences (1 to 32 substeps per interval) and the interpolants (33), rotations on both sides
of one radian, every model's rotation vector, sample blocks and ragged tiles; and the steppers
without a step proposer, whatever proposer the options name."""
import math

import numpy as np
import pytest

from higherharmonics_b200 import api
from tests.helpers import oracle_j, rel_l2

pytestmark = pytest.mark.gpu

# the parity bar of the Magnus-4 tests: the same steps, FP64 rounding only
TOL = 1e-11

SYSTEMS = {
    "dirac2d": (api.SYS_DIRAC2D, dict(velocity=1.0, mass=0.2, pol=(0.6, 0.8))),
    "piflux2d": (api.SYS_PIFLUX2D, dict(hopping=1.0, pol=(0.6, 0.8))),
    "piflux2d_sym": (api.SYS_PIFLUX2D, dict(hopping=1.0, pol=(math.sqrt(0.5), math.sqrt(0.5)))),
    "piflux3d": (api.SYS_PIFLUX3D, dict(hopping=1.0)),
    "honeycomb": (api.SYS_HONEYCOMB, dict(hopping=1.0, mass=0.1, pol=(0.8, 0.6))),
    "honeycomb_x": (api.SYS_HONEYCOMB, dict(hopping=1.0, mass=0.1)),
    "dirac3d": (api.SYS_DIRAC3D, dict()),
}


def _rows(n, seed=5):
    r = np.random.default_rng(seed)
    rows = np.zeros((n, 8))
    rows[:, :3] = r.uniform(0.2, 1.8, (n, 3))
    rows[:, 2] = np.where(r.random(n) < 2, np.hypot(rows[:, 0], rows[:, 1]), 0)
    rows[:, 3] = r.uniform(0.5, 1.0, n)
    s = r.normal(size=(n, 3))
    rows[:, 4:7] = s / np.linalg.norm(s, axis=1, keepdims=True)
    return rows


def _run(engine, name, n_rows=37, n_meas=41, substeps=1, energy=2.0, **kw):
    kind, sk = SYSTEMS[name]
    sys_ = api.system(kind, **sk)
    pulse = api.cosine_pulse(0.8, 1, n_meas, phase=0.4, energy_scale=energy)
    grid, rows = api.grid_explicit(_rows(n_rows))
    opts = api.solver(stepper=api.STEPPER_MAGNUS4, magnus_substeps=substeps, **kw)
    j, st = engine.current_density(sys_, pulse, grid, opts)
    jr, _ = oracle_j(sys_, pulse, rows, 1e-12, 1e-8, stepper=1, magnus_substeps=substeps)
    assert st.attempted_steps == n_rows * n_meas * substeps
    return j, jr


@pytest.mark.parametrize("name", [n for n in SYSTEMS if n != "dirac3d"])
def test_every_model(engine, name):
    j, jr = _run(engine, name)
    assert rel_l2(j, jr) <= TOL


def test_dirac3d_against_rkf78(engine):
    """The oracle has no Magnus-4 step of the Dirac-3D model, so 32 substeps are held to its
    RKF78 solution: 1312 steps of h = 0.0048 with |2 d| <= 4 leave at most 1312 (4 h)^5 / 720 ~
    5e-9."""
    sys_ = api.system(api.SYS_DIRAC3D)
    pulse = api.cosine_pulse(0.8, 1, 41, phase=0.4)
    grid, rows = api.grid_explicit(_rows(37))
    j, _ = engine.current_density(sys_, pulse, grid,
                                  api.solver(stepper=api.STEPPER_MAGNUS4, magnus_substeps=32))
    jr, _ = oracle_j(sys_, pulse, rows, 1e-13, 1e-12)
    assert rel_l2(j, jr) <= 1e-8


@pytest.mark.parametrize("substeps", [1, 2, 3, 32, 33])
@pytest.mark.parametrize("name", ["honeycomb", "piflux2d_sym", "dirac2d"])
def test_substeps(engine, name, substeps):
    j, jr = _run(engine, name, substeps=substeps)
    assert rel_l2(j, jr) <= TOL


@pytest.mark.parametrize("energy", [0.01, 3.0, 12.0, 60.0])
def test_rotation_angles(engine, energy):
    """Angles per interval from 0.005 over one radian (the series' end) to 30."""
    j, jr = _run(engine, "honeycomb_x", energy=energy)
    assert rel_l2(j, jr) <= TOL


@pytest.mark.parametrize("n_rows,n_meas", [(1, 64), (33, 24), (64, 33)])
def test_ragged(engine, n_rows, n_meas):
    j, jr = _run(engine, "piflux2d", n_rows=n_rows, n_meas=n_meas)
    assert rel_l2(j, jr) <= TOL


@pytest.mark.parametrize("substeps", [1, 33])
def test_named_proposer_is_not_read(engine, substeps):
    j, jr = _run(engine, "honeycomb_x", substeps=substeps, proposer=api.PROPOSER_LOCKSTEP)
    assert rel_l2(j, jr) <= TOL
