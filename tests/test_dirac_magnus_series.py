"""The collected rotation vector of the Dirac closed-form Magnus step (struct DiracMagnus of the
device header, compiled here for the host) against the series' nested cross products in exact
rational arithmetic."""
import ctypes
import os
import re
import subprocess
from fractions import Fraction as F

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "higherharmonics_b200", "csrc")


@pytest.fixture(scope="module")
def omega(tmp_path_factory):
    with open(os.path.join(CSRC, "hhg_device.cuh")) as f:
        struct = re.search(r"^struct DiracMagnus \{.*?^\};", f.read(), re.M | re.S).group(0)
    d = tmp_path_factory.mktemp("magnus")
    src = d / "omega.cpp"
    src.write_text("#include <cmath>\nusing std::fma;\n#define __device__\n#define __forceinline__\n"
                   + struct + "\nextern \"C\" void omega(double k_z, double kappa, double mk, double dt,"
                   " const double *m, double *w) { DiracMagnus(k_z, kappa, mk, dt).omega(m, w); }\n")
    lib = d / "omega.so"
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-shared", "-fPIC", str(src), "-o", str(lib)],
                   check=True)
    fn = ctypes.CDLL(str(lib)).omega
    ptr = ctypes.POINTER(ctypes.c_double)
    fn.argtypes = [ctypes.c_double] * 4 + [ptr, ptr]

    def run(k_z, kappa, mk, dt, mom):
        m, w = (ctypes.c_double * 4)(*mom), (ctypes.c_double * 3)()
        fn(k_z, kappa, mk, dt, m, w)
        return list(w)
    return run


def cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def nested(k_z, kappa, mk, dt, mom):
    """MagnusMatrix.cpp:25-57 on axial vectors, every commutator a cross product; the sum and,
    per component, the sum of the terms' sizes (all exact)."""
    k_z, kappa, mk, dt = map(F, (k_z, kappa, mk, dt))
    c = [F(m) / mk for m in mom]
    v = [2 * kappa * dt, F(0), -2 * k_z * dt]
    m1, m2, m3, m4 = ([cq * x for x in v] for cq in c)
    m1[2] += 2 * mk * dt
    c12, c13, c14 = cross(m1, m2), cross(m1, m3), cross(m1, m4)
    c112, c113 = cross(m1, c12), cross(m1, c13)
    terms = [(F(1), m1), (F(-1, 6), c12), (F(-1, 60), cross(m2, c12)), (F(1, 360), cross(m1, c112)),
             (F(1, 140), cross(m2, c14)), (F(-1, 420), cross(m3, c13)), (F(-1, 210), cross(m4, c12)),
             (F(-1, 840), cross(m1, cross(m1, c14))), (F(1, 504), cross(m2, c113)),
             (F(-1, 840), cross(m2, cross(m2, c12))), (F(1, 2520), cross(m3, c112)),
             (F(-1, 2520), cross(m1, cross(m1, c113))), (F(-1, 7560), cross(c12, c112)),
             (F(1, 2520), cross(m2, cross(m1, c112))),
             (F(-1, 15120), cross(m1, cross(m1, cross(m1, c112))))]
    return ([sum(a * t[i] for a, t in terms) for i in range(3)],
            [sum(abs(a * t[i]) for a, t in terms) for i in range(3)])


@pytest.mark.parametrize("scale", [1e-2, 1.0, 8.0])
def test_collected_series(omega, scale):
    """Moments of order |k| (every term enters), angles 2 |k| dt up to a hundredth, one and eight
    radians.  The collected form rounds some 30 operations on numbers no larger than a few times
    the terms' sizes: 100 roundings of their sum."""
    r = np.random.default_rng(int(100 * scale))
    for _ in range(200):
        k_z, kappa = r.uniform(-1.0, 1.0), r.uniform(0.05, 1.0)
        mk = float(np.hypot(k_z, kappa))
        dt = 0.5 * scale * r.uniform(0.1, 1.0) / mk
        mom = mk * r.uniform(-1.0, 1.0, 4)
        w = omega(k_z, kappa, mk, dt, mom)
        exact, size = nested(k_z, kappa, mk, dt, mom)
        for i in range(3):
            assert abs(F(w[i]) - exact[i]) <= 100 * F(2) ** -53 * max(size), (i, w[i], float(exact[i]))
