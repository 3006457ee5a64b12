"""The performance cases of the engine: what a user's program asks of it, through the public
API (higherharmonics_b200.api), from one-shot calls on a small grid to batches of pulses on
the 1024 x 1024 grid.

Five kinds of call:
  oneshot  Engine.current_density + Engine.spectrum: the drop-in for the reference's
           Dispatcher::compute and its FFT, host buffers in and out
  batch    a Plan executed as one graph (integration, Brillouin-zone sum, spectra), then j and
           every spectrum fetched: what bench.py times
  kappa    Engine.dirac_current_density + Engine.spectrum: the Dirac system's adaptive
           momentum quadrature
  kout     Engine.k_resolved: band occupations of every k-point at every sample
  train    Engine.mlp_train: training of the step-size proposer on step histories

Sizes are those of higherharmonics_b200/workloads.py, the tests and the smoke check.  The seed
sets the pulses (amplitude and carrier phase) or the training records.
"""
import math

import numpy as np
import torch

from higherharmonics_b200 import api, workloads

PER_CYCLE = workloads.MEASUREMENTS_PER_CYCLE
# algorithmic flops of one attempted step per k-point (13 right-hand sides and the stage sums)
STEP_FLOPS = {"dirac2d": 577, "piflux2d": 577, "honeycomb": 811, "piflux3d": 577,
              "piflux3d_relax": 1383, "dirac3d_relax": 637}
MAGNUS_FLOPS, DIRAC_MAGNUS_FLOPS = 150, 190
LASER_OMEGA = {"dirac2d": 0.1, "piflux2d": 0.05, "honeycomb": 0.08, "piflux3d": 0.5}


def listed():
    return [
        # the smallest call a program makes: the smoke check's 8 x 8 grid over one cycle,
        # reference schedule, where the latency of the step chain is everything
        dict(name="dirac2d_8", kind="oneshot", model="dirac2d", n1=8, n2=8, cycles=1, pulses=1,
             solver="fp64"),
        # the reference's CPU-sized run: gapped Dirac 64 x 64, 4 cycles, plain FP64 RKF78
        dict(name="dirac2d_64", kind="oneshot", model="dirac2d", n1=64, n2=64, cycles=4, pulses=1,
             solver="fp64"),
        # occupation tracking on the reference's N x N momentum grid (odd N), FP64 RKF78, every
        # k-point's samples back to the host
        dict(name="piflux3d_occupations", kind="kout", model="piflux3d", n1=33, n2=33, cycles=1,
             pulses=1, solver="fp64"),
        # the plain FP64 engine at its ordinary size: pi-flux 256 x 256, 8 cycles
        dict(name="piflux2d_256", kind="batch", model="piflux2d", n1=256, n2=256, cycles=8,
             pulses=1, solver="fp64"),
        # the same grid with FP32 right-hand sides and warp-synchronous steps
        dict(name="piflux2d_256_mixed", kind="batch", model="piflux2d", n1=256, n2=256, cycles=8,
             pulses=1, solver="mixed_lockstep"),
        # the headline workload: honeycomb 1024 x 1024, learned proposer, two pulses of the table
        dict(name="honeycomb_1024_learned", kind="batch", model="honeycomb", n1=1024, n2=1024,
             cycles=6, pulses=2, solver="mixed_learned"),
        # honeycomb 512 x 512 with the Magnus propagator
        dict(name="honeycomb_512_magnus", kind="batch", model="honeycomb", n1=512, n2=512,
             cycles=6, pulses=1, solver="magnus4"),
        # a parameter sweep: pulses of uneven lengths and strengths on 128 x 128 Dirac k-points
        dict(name="dirac2d_sweep_mixed", kind="batch", model="dirac2d", n1=128, n2=128, cycles=0,
             pulses=64, solver="mixed_lockstep"),
        # the reference's production physics (relaxation, 300 K) over one cycle on its
        # continuum-limit grid of 151 552 k-points
        dict(name="piflux3d_relax", kind="oneshot", model="piflux3d_relax", n1=32, n2=4, cycles=1,
             pulses=1, solver="fp64"),
        # the Dirac system's adaptive quadrature, coherent closed-form Magnus step, 8 cycles
        dict(name="dirac3d_kappa", kind="kappa", model="dirac3d", n1=60, n2=100, cycles=8,
             pulses=1, solver="dirac_magnus"),
        # and with relaxation (FP64 RKF78), the path the reference's own configurations take
        dict(name="dirac3d_kappa_relax", kind="kappa", model="dirac3d_relax", n1=60, n2=100,
             cycles=2, pulses=1, solver="fp64"),
        # training of the step-size proposer: 64 batches of 4096 records, two epochs
        dict(name="mlp_train", kind="train", model="mlp", n1=262144, n2=4096, cycles=2, pulses=0,
             solver="adam"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: a kind, then sizes over its whole range."""
    kind = rng.choice(["oneshot", "oneshot", "batch", "batch", "batch", "kout", "kappa", "train",
                       "relax"])
    if kind == "train":
        return dict(kind=kind, model="mlp", n1=_log_int(rng, 20000, 500000),
                    n2=128 * rng.choice([8, 16, 32, 33, 64]), cycles=rng.choice([1, 2]), pulses=0,
                    solver="adam")
    if kind == "kappa":
        relax = rng.random() < 0.4
        return dict(kind=kind, model="dirac3d_relax" if relax else "dirac3d",
                    n1=rng.randint(9, 60), n2=rng.randint(20, 100),
                    cycles=rng.choice([1, 2]) if relax else rng.randint(2, 8), pulses=1,
                    solver="fp64" if relax else "dirac_magnus")
    if kind == "relax":
        return dict(kind="oneshot", model="piflux3d_relax", n1=rng.randint(5, 32),
                    n2=rng.choice([2, 3, 4]), cycles=1, pulses=1, solver="fp64")
    if kind == "kout":
        return dict(kind=kind, model="piflux3d", n1=2 * rng.randint(5, 24) + 1, n2=0,
                    cycles=rng.choice([1, 2]), pulses=1, solver="fp64")
    model = rng.choice(["dirac2d", "piflux2d", "honeycomb"])
    if kind == "oneshot":
        return dict(kind=kind, model=model, n1=_log_int(rng, 5, 120), n2=_log_int(rng, 5, 120),
                    cycles=rng.randint(1, 6), pulses=1,
                    solver=rng.choice(["fp64", "fp64", "magnus4"]))
    solver = rng.choice(["fp64", "mixed_lockstep", "mixed_lockstep", "magnus4", "mixed_learned"])
    if solver == "mixed_learned":
        model = "honeycomb"
    n1 = _log_int(rng, 64, 360)
    return dict(kind=kind, model=model, n1=n1, n2=_log_int(rng, 64, 360),
                cycles=rng.randint(2, 8), pulses=rng.choice([1, 1, 2, 3]) if n1 < 250 else 1,
                solver=solver)


# ---------------------------------------------------------------------------
# the call's inputs
# ---------------------------------------------------------------------------
def _system(case):
    model = case["model"]
    if model == "dirac2d":
        return api.system(api.SYS_DIRAC2D, velocity=1.0, mass=0.05)
    if model == "piflux2d":
        s = 1.0 / math.sqrt(2.0)
        return api.system(api.SYS_PIFLUX2D, hopping=1.0, pol=(s, s))
    if model == "honeycomb":
        return api.system(api.SYS_HONEYCOMB, hopping=1.0, mass=0.1)
    return api.system(api.SYS_PIFLUX3D, hopping=1.0)


def _pulse_parameters(case, seed):
    """(amplitude, cycles, intervals, window end, phase, energy scale) of every pulse."""
    r = np.random.default_rng(seed)
    lengths = np.random.default_rng(case["pulses"])  # a sweep's lengths are its own, not the seed's
    out = []
    for _ in range(case["pulses"]):
        omega = LASER_OMEGA[case["model"]]
        cycles = case["cycles"]
        if case["model"] == "honeycomb":
            amplitude, phase = r.uniform(0.5, 2.0), r.uniform(0.0, 2 * math.pi)
        elif cycles == 0:  # the sweep's pulses
            amplitude = math.exp(r.uniform(math.log(0.1), math.log(2.0)))
            phase = r.uniform(0.0, 2 * math.pi)
            cycles, omega = lengths.uniform(2.0, 10.0), lengths.uniform(0.05, 0.15)
        else:
            amplitude, phase = r.uniform(0.8, 1.2), r.uniform(0.0, 2 * math.pi)
        tail = 0 if case["model"] == "dirac2d" else 1  # the lattice models' relaxation cycle
        out.append((amplitude, cycles, int(round(PER_CYCLE * cycles)),
                    2 * math.pi * (cycles + tail), phase, 1.0 / omega))
    return out


def _grid(case):
    n1, n2 = case["n1"], case["n2"]
    if case["kind"] == "kout":
        return api.grid_piflux3d_occupation(n1)
    if case["model"] == "dirac2d":
        return api.grid_tensor(n1, n2, -2, 2, -2, 2)
    if case["model"] == "piflux2d":
        return api.grid_tensor(n1, n2, -math.pi, math.pi, -math.pi, math.pi)
    return api.grid_rhombic(n1, n2)


def _records(n, seed):
    """Step histories as learned_collect writes them: momenta over the zone, A and E of a pulse,
    Bloch vectors, the previous level, and the level the error norm would accept."""
    r = np.random.default_rng(seed)
    rec = np.zeros((n, api.HIST_FIELDS), np.float32)
    rec[:, 0:2] = r.uniform(-1, 1, (n, 2))
    rec[:, 2:4] = r.uniform(-2, 2, (n, 2))
    s = r.normal(size=(n, 3))
    rec[:, 4:7] = s / np.linalg.norm(s, axis=1, keepdims=True)
    rec[:, 7] = -r.integers(0, 4, n)
    rec[:, 8] = (-0.7 + 0.25 * np.cos(math.pi * rec[:, 0]) + 0.15 * np.abs(rec[:, 3]) +
                 0.1 * rec[:, 4] + 0.05 * r.normal(size=n))
    rec[:, 9] = 2.0 ** rec[:, 7]
    return rec


def _solver(case, seed):
    name = case["solver"]
    tol = dict(abs_tol=1e-12, rel_tol=1e-8)
    if case["model"] == "dirac2d":
        tol = dict(abs_tol=1e-10, rel_tol=1e-10)
    if name == "magnus4":
        return api.solver(stepper=api.STEPPER_MAGNUS4, **tol)
    if name == "dirac_magnus":
        return api.solver(stepper=api.STEPPER_DIRAC_MAGNUS, **tol)
    if name == "fp64":
        return api.solver(**tol)
    mixed = dict(abs_tol=1e-8, rel_tol=1e-6, precision=api.PREC_MIXED)
    if name == "mixed_lockstep":
        return api.solver(proposer=api.PROPOSER_LOCKSTEP, **mixed)
    return api.solver(proposer=api.PROPOSER_LEARNED, mlp=api.mlp_init(1, _records(4096, seed)),
                      **mixed)


def prepare(case, seed):
    eng = api.Engine(0)
    s = {"case": case, "eng": eng}
    if case["kind"] == "train":
        s["records"] = _records(case["n1"], seed)
        s["net"] = api.mlp_init(1 + seed % 1000, s["records"])
        s["opts"] = api.train_opts(epochs=case["cycles"], batch=case["n2"], seed=seed)
        return s
    s["opts"] = _solver(case, seed)
    if case["kind"] == "kappa":
        w = workloads.dirac3d_kappa(case["cycles"], relax=case["model"] == "dirac3d_relax")
        r = np.random.default_rng(seed)
        w.pulse.amplitude *= r.uniform(0.9, 1.1)
        w.pulse.phase = r.uniform(0.0, 2 * math.pi)
        s["system"], s["pulses"] = w.system, [w.pulse]
        s["quad"] = api.kappa_quad(w.quad.max_k, case["n1"], w.quad.n_kappa, w.quad.threshold,
                                   case["n2"])
        return s
    if case["model"] == "piflux3d_relax":
        w = workloads.piflux3d_relax(case["cycles"])
        r = np.random.default_rng(seed)
        w.pulses[0].amplitude *= r.uniform(0.9, 1.1)
        s["system"], s["pulses"] = w.system, w.pulses
        s["grid"] = api.grid_piflux3d_ref(case["n1"], case["n2"])
        return s
    s["system"], s["grid"] = _system(case), _grid(case)
    s["pulses"] = [api.cosine_pulse(a, c, n, phase=ph, window=(0.0, end), energy_scale=es)
                   for a, c, n, end, ph, es in _pulse_parameters(case, seed)]
    if case["kind"] == "batch":
        s["plan"] = eng.plan(s["system"], s["pulses"], s["grid"], s["opts"])
    return s


def run(s):
    kind = s["case"]["kind"]
    eng = s["eng"]
    if kind == "train":
        net = api.Mlp.from_buffer_copy(s["net"])
        loss, _ = eng.mlp_train(s["records"], net, s["opts"])
        return {"params": net.param_array().copy(), "loss": loss}
    if kind == "batch":
        plan = s["plan"]
        plan.execute_graph()
        j, _ = plan.fetch()
        spectra = [plan.fetch_spectrum(p) for p in range(len(s["pulses"]))]
        return {"j": j, "freq": np.concatenate([f for f, _, _ in spectra]),
                "re": np.concatenate([a for _, a, _ in spectra]),
                "im": np.concatenate([b for _, _, b in spectra])}
    p = s["pulses"][0]
    if kind == "kout":
        occ, _ = eng.k_resolved(s["system"], p, s["grid"], s["opts"], api.KOUT_OCCUPATIONS)
        return {"occupations": occ}
    if kind == "kappa":
        j, _, _ = eng.dirac_current_density(s["system"], p, s["quad"], s["opts"])
    else:
        j, _ = eng.current_density(s["system"], p, s["grid"], s["opts"])
    fr, re, im = eng.spectrum(j, p.n_measurements, p.window_begin, p.window_end)
    return {"j": j, "freq": fr, "re": re, "im": im}


def _n_k(case):
    if case["model"] == "piflux3d_relax":
        c = case["n2"]
        return 2 * case["n1"] * (128 * c * c + 12 * c * c + 8 * c * c)
    if case["kind"] == "kout":
        return case["n1"] * case["n1"]
    return case["n1"] * case["n2"]


def work(case):
    if case["kind"] == "train":
        # forward and backward of the four layers, the records read once per epoch
        rows = case["n1"] // min(case["n2"], case["n1"]) * min(case["n2"], case["n1"])
        return {"bytes": 48.0 * case["n1"] * case["cycles"],
                "flops": 6.0 * rows * case["cycles"] * (8 * 64 + 2 * 64 * 64 + 64)}
    if case["kind"] == "kappa":
        n = PER_CYCLE * case["cycles"]
        nodes = (case["n1"] - 2) * case["n2"] * 21.0
        per = 4 * STEP_FLOPS["dirac3d_relax"] if case["solver"] == "fp64" else DIRAC_MAGNUS_FLOPS
        return {"bytes": 8.0 * (9 * n + 8 * nodes), "flops": nodes * n * per}
    n_k = _n_k(case)
    if case["cycles"] == 0:
        samples = case["pulses"] * 6 * PER_CYCLE  # cycles uniform in [2, 10]
    else:
        samples = case["pulses"] * case["cycles"] * PER_CYCLE
    if case["solver"] == "magnus4":
        per = MAGNUS_FLOPS
    else:
        # reference schedule: four steps an interval (five with relaxation); dyadic: one
        steps = 5 if case["model"] == "piflux3d_relax" else 4 if case["solver"] == "fp64" else 1
        per = steps * STEP_FLOPS[case["model"]]
    out = 16.0 * n_k * samples if case["kind"] == "kout" else 8.0 * 13 * samples
    return {"bytes": 64.0 * n_k + out, "flops": float(per) * n_k * samples}


# ---------------------------------------------------------------------------
# the same values in 64 bits: sixth-order Magnus steps of dS/dt = 2 d(k - A(t)) x S, four per
# sampling interval, and the trapezoidal Fourier sum, in torch and numpy
# ---------------------------------------------------------------------------
SUBSTEPS = 4
CHUNK = 8  # intervals whose rotations are formed at once


def _gl(n, lo, hi):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (hi - lo) * x + 0.5 * (hi + lo), 0.5 * (hi - lo) * w


def _points(case):
    """kx, ky, weights of the case's grid."""
    if case["model"] == "honeycomb":
        f1, w1 = _gl(case["n1"], -0.5, 0.5)
        f2, w2 = _gl(case["n2"], -0.5, 0.5)
        a, b = 2 * math.pi / 3, 2 * math.pi / math.sqrt(3.0)
        F1, F2 = np.meshgrid(f1, f2, indexing="ij")
        return a * (F1 + F2), b * (F2 - F1), np.outer(w1, w2) * 2 * a * b
    lim = 2.0 if case["model"] == "dirac2d" else math.pi
    x, wx = _gl(case["n1"], -lim, lim)
    y, wy = _gl(case["n2"], -lim, lim)
    return *np.meshgrid(x, y, indexing="ij"), np.outer(wx, wy)


def _field(par, t):
    a, c, _, _, ph, _ = par
    inside = (t > 0.0) & (t < 2 * math.pi * c)
    return np.where(inside, a * 0.5 * (1 - np.cos(t / c)) * np.sin(t + ph), 0.0)


def _linear_form(case, kx, ky, es):
    """D, V, functions: d(k - A) = D . f(A), the vertex vector V . f(A), f a list of functions."""
    dev = kx.device
    n = kx.shape[0]
    one, zero = torch.ones(n, dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev)
    if case["model"] == "dirac2d":
        D = torch.stack([torch.stack([es * kx, -es * one]), torch.stack([es * ky, zero]),
                         torch.stack([0.05 * es * one, zero])])
        V = torch.stack([torch.stack([one, zero]), torch.stack([zero, zero]),
                         torch.stack([zero, zero])])
        return D, V, [np.ones_like, lambda A: A]
    if case["model"] == "piflux2d":
        p = 1.0 / math.sqrt(2.0)
        D = -2 * es * torch.stack([torch.stack([kx.cos(), kx.sin()]), torch.stack([ky.cos(), ky.sin()]),
                                   torch.stack([zero, zero])])
        V = p * torch.stack([torch.stack([kx.sin(), -kx.cos()]), torch.stack([ky.sin(), -ky.cos()]),
                             torch.stack([zero, zero])])
        return D, V, [lambda A: np.cos(p * A), lambda A: np.sin(p * A)]
    h = 0.5 * math.sqrt(3.0)
    b1, b2, b3 = kx, -0.5 * kx + h * ky, -0.5 * kx - h * ky
    c1, s1, c2, s2 = b1.cos(), b1.sin(), b2.cos() + b3.cos(), b2.sin() + b3.sin()
    # gamma = e^{i b1 - iA} + (e^{i b2} + e^{i b3}) e^{iA/2}; f = cos A, sin A, cos A/2, sin A/2, 1
    D = es * torch.stack([torch.stack([c1, s1, c2, -s2, zero]), -torch.stack([s1, -c1, s2, c2, zero]),
                          torch.stack([zero, zero, zero, zero, 0.1 * one])])
    V = torch.stack([torch.stack([c1, s1, -0.5 * c2, 0.5 * s2, zero]),
                     torch.stack([s1, -c1, -0.5 * s2, -0.5 * c2, zero]),
                     torch.zeros(5, n, dtype=torch.float64, device=dev)])
    return D, V, [np.cos, np.sin, lambda A: np.cos(0.5 * A), lambda A: np.sin(0.5 * A), np.ones_like]


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _exact_current(case, par, dev):
    _, _, N, end, _, es = par
    kx, ky, w = (torch.tensor(np.ascontiguousarray(v).reshape(-1), dtype=torch.float64, device=dev)
                 for v in _points(case))
    D, V, fs = _linear_form(case, kx, ky, es)
    # j = sum_k w (V . f(A)) . S, the model vertex
    S = -torch.einsum("cfn,f->cn", D, torch.tensor([float(f(np.zeros(1))[0]) for f in fs],
                                                   dtype=torch.float64, device=dev))
    S = S / S.norm(dim=0)
    dt = end / N
    h = dt / SUBSTEPS
    g = math.sqrt(15.0) / 10.0
    starts = (np.arange(N * SUBSTEPS) * h)[:, None] + h * np.array([0.5 - g, 0.5, 0.5 + g])
    F = torch.tensor(np.stack([f(_field(par, starts)) for f in fs]), device=dev)  # (f, step, 3)
    G = torch.tensor(np.stack([f(_field(par, np.arange(N + 1) * dt)) for f in fs]), device=dev)
    j = torch.zeros(N + 1, dtype=torch.float64, device=dev)

    def sample(i):
        j[i] = (w * (torch.einsum("cfn,f->cn", V, G[:, i]) * S).sum(0)).sum()

    sample(0)
    for i0 in range(0, N, CHUNK):
        i1 = min(N, i0 + CHUNK)
        d = 2 * h * torch.einsum("cfn,fsg->gcsn", D, F[:, i0 * SUBSTEPS:i1 * SUBSTEPS])
        a1, a2, a3 = d[1], math.sqrt(15.0) / 3 * (d[2] - d[0]), 10.0 / 3 * (d[2] - 2 * d[1] + d[0])
        c1 = _cross(a1, a2)
        c2 = -_cross(a1, 2 * a3 + c1) / 60
        om = a1 + a3 / 12 + _cross(-20 * a1 - a3 + c1, a2 + c2) / 240
        th = om.square().sum(0).sqrt().clamp_min(1e-30)
        sa, ca = th.sin() / th, 2 * ((0.5 * th).sin() / th).square()
        for q in range(om.shape[1]):
            o = om[:, q]
            u = _cross(o, S)
            S = S + sa[q] * u + ca[q] * _cross(o, u)
            if (q + 1) % SUBSTEPS == 0:
                sample(i0 + (q + 1) // SUBSTEPS)
    return j.cpu().numpy()


def _exact_spectrum(j, N, end):
    n_in = 8 * (N + 1)
    x = np.concatenate([j, np.zeros(n_in - j.size)])
    dt = end / N
    fr = 2 * np.pi * np.arange(n_in // 2 + 1) / (n_in * dt)
    th = fr * dt
    small = np.abs(th) < 1e-12
    t = np.where(small, 1.0, th)
    W = np.where(small, 1.0, 2 * (1 - np.cos(t)) / t ** 2)
    a0 = np.where(small, -0.5, -(1 - np.cos(t)) / t ** 2 + 1j * (t - np.sin(t)) / t ** 2)
    out = dt * (dt * W * np.fft.rfft(x) + a0 * x[0])
    return fr, out.real, out.imag


def exact(case, seed):
    # no 64-bit value: the relaxation runs depend on the reference's step sequence, the adaptive
    # quadrature on its refinement, training on the rounding of BF16 weights along the way; the
    # largest batches and the occupation grids take too long
    if case["kind"] not in ("oneshot", "batch") or case["model"] == "piflux3d_relax":
        return None
    pars = _pulse_parameters(case, seed)
    if case["n1"] * case["n2"] * sum(p[2] for p in pars) > 6e8 or sum(p[2] for p in pars) > 9000:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    js = [_exact_current(case, p, dev) for p in pars]
    spectra = [_exact_spectrum(j, p[2], p[3]) for j, p in zip(js, pars)]
    return {"j": np.concatenate(js), "freq": np.concatenate([s[0] for s in spectra]),
            "re": np.concatenate([s[1] for s in spectra]),
            "im": np.concatenate([s[2] for s in spectra])}
