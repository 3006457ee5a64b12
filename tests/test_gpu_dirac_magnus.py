"""GPU checks of the closed-form Dirac Magnus step where its rotation takes another form: angles
per interval below 2, between 2 and 4, above 4, and all of them in one warp, in a field strong
enough that every Legendre moment of the interval enters; and a trajectory's independence of the
rows that share its warp."""
import math

import numpy as np
import pytest

from higherharmonics_b200 import api
from tests.helpers import oracle_j, rel_l2

pytestmark = pytest.mark.gpu

N_MEAS = 96
# |k| for an angle of 2 |k| dt a radian: the field moves it by some tenths
PER_RADIAN = N_MEAS / (4 * math.pi)
ANGLES = {"below_2": (0.2, 1.5), "2_to_4": (2.4, 3.4), "above_4": (4.6, 9.0), "mixed": (0.2, 9.0)}


def _rows(lo, hi, n=40, seed=3):
    r = np.random.default_rng(seed)
    k = PER_RADIAN * np.linspace(lo, hi, n)
    r.shuffle(k)
    phi = r.uniform(0.2, math.pi - 0.2, n)
    rows = np.zeros((n, 8))
    rows[:, 0], rows[:, 1] = k * np.cos(phi), k * np.sin(phi)
    rows[:, 2] = np.hypot(rows[:, 0], rows[:, 1])
    rows[:, 3] = r.uniform(0.5, 1.0, n)
    rows[:, 6] = -1.0
    return rows


def _pulse():
    # A up to 3 over |k| of 1.5 and more: the moments cf_q = m_q / |k| reach 2, 0.2, 0.01, ...
    return api.cosine_pulse(3.0, 1, N_MEAS, phase=0.7)


# One step per interval without step control: product and oracle differ by rounding.  A step's
# rotation vector and factors carry some 30 rounded operations each, so a state moves by at most
# about 60 x 1.1e-16 x max(1, angle / 2) an interval: 96 x 60 x 1.1e-16 x 4.5 = 2.9e-12 in the
# worst case of all errors in one direction, a tenth of it as a sum of random signs.
TOL = 3e-12


@pytest.mark.parametrize("name", list(ANGLES))
def test_matches_oracle(engine, name):
    rows, sys_, pulse = _rows(*ANGLES[name]), api.system(api.SYS_DIRAC3D), _pulse()
    grid, _ = api.grid_explicit(rows)
    j, st = engine.current_density(sys_, pulse, grid, api.solver(stepper=api.STEPPER_DIRAC_MAGNUS))
    jr, _ = oracle_j(sys_, pulse, rows, 1e-12, 1e-8, stepper=2)
    assert st.attempted_steps == len(rows) * N_MEAS and st.failed_trajectories == 0
    assert rel_l2(j, jr) <= TOL, rel_l2(j, jr)


def test_trajectories_do_not_depend_on_their_warp(engine):
    sys_, pulse = api.system(api.SYS_DIRAC3D), _pulse()
    opts = api.solver(stepper=api.STEPPER_DIRAC_MAGNUS)

    def run(rows):
        grid, _ = api.grid_explicit(np.ascontiguousarray(rows))
        return engine.k_resolved(sys_, pulse, grid, opts, api.KOUT_CURRENT)[0]

    rows = _rows(*ANGLES["mixed"])
    order = np.argsort(rows[:, 2])
    together, by_size = run(rows), run(rows[order])
    assert np.array_equal(together[:, order], by_size)
    assert all(np.array_equal(together[:, q], run(rows[q:q + 1])[:, 0]) for q in range(0, 40, 7))
