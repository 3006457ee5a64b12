"""GPU checks of small grids run with their intervals in parallel (chunks of intervals from the
propagators before them) against the sequential run of the same plan (tile_k = 2 asks for two
tiles per item, which runs sequentially): every coherent model, both steppers, uneven pulses,
ragged rows, the k-resolved outputs, runs that leave the standard schedule (the chunked run is
discarded), failures, repeated executions and graph launches."""
import math

import numpy as np
import pytest

from higherharmonics_b200 import api
from tests.helpers import oracle_j, rel_l2
from tests.test_gpu_magnus_table import SYSTEMS, _rows

pytestmark = pytest.mark.gpu

# rounding of the chunks' start states (1e-11 of |S| is where a chunk is refused; the sums of
# propagated rounding over a few hundred intervals stay below 1e-13)
TOL = 1e-12


def _both(engine, name, pulses, n_rows=40, **kw):
    kind, sk = SYSTEMS[name]
    sys_ = api.system(kind, **sk)
    grid, rows = api.grid_explicit(_rows(n_rows))
    j, st = engine.current_density(sys_, pulses, grid, api.solver(**kw))
    js, ss = engine.current_density(sys_, pulses, grid, api.solver(tile_k=2, **kw))
    return sys_, rows, j, st, js, ss


@pytest.mark.parametrize("name", list(SYSTEMS))
@pytest.mark.parametrize("stepper", [api.STEPPER_RKF78, api.STEPPER_MAGNUS4])
def test_matches_sequential(engine, name, stepper):
    p = api.cosine_pulse(0.7, 1, 333, phase=0.3, energy_scale=4.0)
    sys_, rows, j, st, js, ss = _both(engine, name, p, stepper=stepper)
    assert rel_l2(j, js) <= TOL
    assert st.attempted_steps == ss.attempted_steps and st.rejected_steps == ss.rejected_steps
    if stepper == api.STEPPER_RKF78:
        jr, _ = oracle_j(sys_, p, rows, 1e-12, 1e-8)
        assert rel_l2(j, jr) <= 1e-9


@pytest.mark.parametrize("n_rows", [1, 31, 33, 200])
@pytest.mark.parametrize("n_meas", [63, 64, 65, 71, 72, 73, 520])
def test_edges(engine, n_rows, n_meas):
    p = api.cosine_pulse(0.7, 1, n_meas, energy_scale=2.0 * n_meas / 100)
    _, _, j, st, js, ss = _both(engine, "honeycomb_x", p, n_rows)
    assert rel_l2(j, js) <= TOL and st.attempted_steps == ss.attempted_steps


@pytest.mark.parametrize("stepper,substeps", [(api.STEPPER_RKF78, 1), (api.STEPPER_MAGNUS4, 3)])
def test_uneven_pulses(engine, stepper, substeps):
    pulses = [api.cosine_pulse(0.3 + 0.2 * i, 1 + 0.3 * i, n, phase=i, energy_scale=3.0,
                               window=(0.0, 2 * math.pi * n / 200))
              for i, n in enumerate([400, 65, 7, 129, 256])]
    _, _, j, st, js, ss = _both(engine, "dirac2d", pulses, stepper=stepper, magnus_substeps=substeps)
    assert rel_l2(j, js) <= TOL and st.attempted_steps == ss.attempted_steps


@pytest.mark.parametrize("energy", [40.0, 200.0])
def test_off_schedule_runs_are_discarded(engine, energy):
    """Rejections and steps below the schedule's: the sequential run stands, bit for bit."""
    p = api.cosine_pulse(0.7, 1, 200, energy_scale=energy)
    _, _, j, st, js, ss = _both(engine, "honeycomb_x", p, n_rows=32)
    assert ss.attempted_steps > 4 * 32 * 200
    assert st.attempted_steps == ss.attempted_steps and rel_l2(j, js) <= 1e-15


def test_failures_are_reported(engine):
    kind, sk = SYSTEMS["honeycomb_x"]
    p = api.cosine_pulse(0.7, 1, 200, energy_scale=200.0)
    grid, _ = api.grid_explicit(_rows(8))
    opts = api.solver(1e-14, 1e-14)
    opts.max_attempts_per_interval = 2
    with pytest.raises(api.HHGError) as e:
        engine.current_density(api.system(kind, **sk), p, grid, opts)
    assert e.value.status == api.STEP_LIMIT


@pytest.mark.parametrize("kind", [api.KOUT_BLOCH, api.KOUT_OCCUPATIONS])
def test_k_resolved(engine, kind):
    sys_ = api.system(api.SYS_PIFLUX3D, hopping=2.0, beta=0.3, fermi_energy=0.4)
    p = api.cosine_pulse(0.7, 1, 250, energy_scale=1.0)
    grid = api.grid_piflux3d_occupation(9)
    out, st = engine.k_resolved(sys_, p, grid, api.solver(), kind)
    seq, ss = engine.k_resolved(sys_, p, grid, api.solver(tile_k=2), kind)
    assert st.attempted_steps == ss.attempted_steps
    assert np.max(np.abs(out - seq)) <= 1e-9  # occupations: a root of a difference near 0


def test_repeated_and_graph(engine):
    kind, sk = SYSTEMS["piflux2d"]
    p = api.cosine_pulse(0.7, 1, 300, energy_scale=2.0)
    grid, _ = api.grid_explicit(_rows(50))
    plan = engine.plan(api.system(kind, **sk), p, grid, api.solver())
    runs = []
    for graph in (False, False, True, True):
        plan.execute_graph() if graph else plan.execute_async()
        j, st = plan.fetch()
        runs.append((j, st.attempted_steps))
    plan.close()
    assert all(np.array_equal(j, runs[0][0]) and a == runs[0][1] for j, a in runs)


def test_batches_agree_with_single_runs(engine):
    """Up to one tile per SM in the whole batch: bit for bit."""
    sys_ = api.system(api.SYS_DIRAC2D, velocity=1.0, mass=0.05)
    pulses = [api.cosine_pulse(0.3 + 0.1 * i, 1.5, 512 + 200 * i, phase=0.4 * i, energy_scale=8.0)
              for i in range(6)]
    grid = api.grid_tensor(24, 24, -2, 2, -2, 2)
    jb, _ = engine.current_density(sys_, pulses, grid, api.solver(1e-10, 1e-10))
    single = [engine.current_density(sys_, p, grid, api.solver(1e-10, 1e-10))[0] for p in pulses]
    assert np.array_equal(jb, np.concatenate(single))
