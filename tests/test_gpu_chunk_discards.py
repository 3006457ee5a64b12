"""GPU checks of chunked runs that are discarded: in a batch beside a pulse that stands, at a
chunk's end alone (every error inside the schedule's bounds for a state of length one, the rows'
states longer), executed again and as a graph; the batch beyond one tile per SM; and the price of
a discarded run, paid by a plan's first execution only."""
import math

import numpy as np
import pytest

from higherharmonics_b200 import api
from tests.helpers import rel_l2
from tests.test_gpu_magnus_table import SYSTEMS, _rows

pytestmark = pytest.mark.gpu

# chunked against sequential: rounding of the chunks' start states (a chunk is refused at 1e-12
# of |S|)
TOL = 1e-12


def _system(name):
    kind, sk = SYSTEMS[name]
    return api.system(kind, **sk)


def _runs(engine, sys_, pulses, grid, opts, graphs=(False, False, True)):
    plan = engine.plan(sys_, pulses, grid, opts)
    out = []
    for graph in graphs:
        plan.execute_graph() if graph else plan.execute_async()
        j, st = plan.fetch()
        out.append((j, st.attempted_steps, st.rejected_steps, st.kernel_ms))
    plan.close()
    return out


def test_one_of_a_batch(engine):
    pulses = [api.cosine_pulse(0.7, 1, 200, phase=0.3, energy_scale=es) for es in (4.0, 40.0, 3.0)]
    grid, _ = api.grid_explicit(_rows(32))
    runs = _runs(engine, _system("honeycomb_x"), pulses, grid, api.solver())
    seq = _runs(engine, _system("honeycomb_x"), pulses, grid, api.solver(tile_k=2), (False,))[0]
    part = [slice(201 * p, 201 * (p + 1)) for p in range(3)]
    assert seq[1] > 4 * 32 * 600  # the second pulse leaves the schedule
    for j, attempts, rejects, _ in runs:
        assert np.array_equal(j, runs[0][0]) and (attempts, rejects) == seq[1:3]
        assert np.array_equal(j[part[1]], seq[0][part[1]])
        assert rel_l2(j[part[0]], seq[0][part[0]]) <= TOL
        assert rel_l2(j[part[2]], seq[0][part[2]]) <= TOL


def test_at_a_chunks_end(engine):
    """States of length 100 under an absolute tolerance: they leave the schedule at a hundredth of
    the error that a state of length one may have, which the propagators' bounds allow, and their
    chunks end 7e-9 of |S| from the propagators (the oracle's runs of both lengths)."""
    rows = _rows(32)
    rows[:, 4:7] *= 100.0
    grid, _ = api.grid_explicit(rows)
    p = api.cosine_pulse(0.7, 1, 160, phase=0.3, energy_scale=4.0)
    opts = dict(abs_tol=1e-7, rel_tol=0.0)
    seq = _runs(engine, _system("honeycomb_x"), [p], grid, api.solver(tile_k=2, **opts), (False,))[0]
    assert seq[1] > 4 * 32 * 160
    for j, attempts, rejects, _ in _runs(engine, _system("honeycomb_x"), [p], grid, api.solver(**opts)):
        assert np.array_equal(j, seq[0]) and (attempts, rejects) == seq[1:3]


def test_batch_beyond_one_tile_per_sm(engine):
    """The batch runs sequentially, its pulses' single runs in chunks: equal up to rounding."""
    sys_ = api.system(api.SYS_DIRAC2D, velocity=1.0, mass=0.05)
    pulses = [api.cosine_pulse(0.3 + 0.1 * i, 1.5, 512, phase=0.4 * i, energy_scale=8.0) for i in range(4)]
    grid, opts = api.grid_tensor(48, 48, -2, 2, -2, 2), api.solver(1e-10, 1e-10)
    jb, _ = engine.current_density(sys_, pulses, grid, opts)
    for p, j in zip(pulses, np.split(jb, 4)):
        assert rel_l2(j, engine.current_density(sys_, p, grid, opts)[0]) <= TOL


def test_price_is_paid_once(engine):
    """128 tiles whose chunks disagree at their ends only, the dearest discard there is (1.6 times
    the sequential run): later executions go straight to the sequential run."""
    sys_ = api.system(api.SYS_HONEYCOMB, hopping=1.0, mass=0.1)
    p = api.cosine_pulse(1.0, 2, 2048, energy_scale=28.0)
    grid = api.grid_rhombic(64, 64)
    _runs(engine, sys_, [p], grid, api.solver())  # (first launches load the kernels)
    ms = [r[3] for r in _runs(engine, sys_, [p], grid, api.solver(), (False,) * 4)]
    assert min(ms[1:]) <= 0.85 * ms[0], ms
