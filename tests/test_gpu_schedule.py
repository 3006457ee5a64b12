"""GPU checks of the standard-schedule path against the oracle, at the sizes where its pieces
end: sample blocks of eight (n_measurements around multiples of 8), one interval, ragged and
single k rows, several tiles per item, schedules of one to five and of more tabulated steps
(n_subdivisions), and tolerances that take lanes off the schedule on every step."""
import math

import numpy as np
import pytest

from higherharmonics_b200 import api
from oracle import hhg_oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

# j(t) within the plain FP64 bar of the parity tests
TOL = 1e-9


def _case(n_meas, n_sub, tol, n1=5, n2=7, tile_k=0, model="honeycomb"):
    cyc = 1
    end = 2 * math.pi * n_meas / 256
    if model == "honeycomb":
        sys_ = api.system(api.SYS_HONEYCOMB, hopping=1.0, mass=0.1)
        m = O.model(O.HONEYCOMB, hopping=5.0, mass=0.5)
        grid = api.grid_rhombic(n1, n2)
    else:
        sys_ = api.system(api.SYS_DIRAC2D, velocity=1.0, mass=0.05)
        m = O.model(O.DIRAC2D, velocity=5.0, mass=0.25)
        grid = api.grid_tensor(n1, n2, -2, 2, -2, 2)
    p = api.cosine_pulse(0.9, cyc, n_meas, phase=0.7, window=(0.0, end), energy_scale=5.0,
                         n_subdivisions=n_sub)
    rows = api.grid_rows(sys_, grid)
    jr, st, rc = O.current_density(m, O.Pulse(0.9, cyc, phase=0.7),
                                   O.time_config(0.0, end, n_meas, n_sub), O.solver(*tol), rows)
    assert rc == 0
    return sys_, p, grid, api.solver(*tol, tile_k=tile_k), jr, st


@pytest.mark.parametrize("n_meas", [1, 7, 8, 9, 63, 65])
def test_sample_blocks(engine, n_meas):
    sys_, p, grid, opts, jr, _ = _case(n_meas, 50, (1e-12, 1e-8))
    j, _ = engine.current_density(sys_, p, grid, opts)
    assert np.all(np.isfinite(j)) and rel_l2(j, jr) <= TOL


@pytest.mark.parametrize("n1,n2,tile_k", [(1, 1, 0), (1, 33, 0), (9, 11, 2), (13, 17, 3)])
def test_ragged_tiles(engine, n1, n2, tile_k):
    sys_, p, grid, opts, jr, _ = _case(20, 50, (1e-12, 1e-8), n1, n2, tile_k, "dirac2d")
    j, _ = engine.current_density(sys_, p, grid, opts)
    assert rel_l2(j, jr) <= TOL


@pytest.mark.parametrize("n_sub", [1, 2, 5, 50, 3000, 100000])
@pytest.mark.parametrize("tol", [(1e-12, 1e-8), (1e-13, 1e-12), (1e-5, 1e-4)])
def test_schedules(engine, n_sub, tol):
    """One to five tabulated steps and beyond; loose and tight tolerances (on and off it)."""
    sys_, p, grid, opts, jr, st_o = _case(24, n_sub, tol)
    j, st = engine.current_density(sys_, p, grid, opts)
    # the step sequence is the oracle's, so is j to the rounding of its steps: at loose
    # tolerances a decision on a threshold may differ and then moves j by the tolerance
    assert rel_l2(j, jr) <= max(TOL, 0.01 * tol[1])
    assert abs(st.attempted_steps - st_o.attempted) <= 2e-3 * st_o.attempted


@pytest.mark.parametrize("precision,n_meas", [(api.PREC_FP64, n) for n in (1, 7, 8, 9, 17, 64)] +
                         [(api.PREC_MIXED, n) for n in (7, 8, 9, 17, 64)])
@pytest.mark.parametrize("model", ["honeycomb", "dirac2d"])
def test_dyadic_sample_blocks(engine, model, precision, n_meas):
    """The dyadic steppers' blocks and records (rel_tol 1e-8; FP32 stages: 6e-8 of the
    trajectories' size a step, so the mixed runs start at windows whose current has risen to
    more than a millionth of it)."""
    sys_, p, grid, _, jr, _ = _case(n_meas, 50, (1e-12, 1e-8), 9, 5, model=model)
    j, _ = engine.current_density(sys_, p, grid,
                                  api.solver(1e-12, 1e-8, precision=precision,
                                             proposer=api.PROPOSER_LOCKSTEP))
    bar = 1e-7 if precision == api.PREC_FP64 else 1e-5
    assert np.all(np.isfinite(j)) and rel_l2(j, jr) <= bar
