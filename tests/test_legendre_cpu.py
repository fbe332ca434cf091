"""The explicit Legendre polynomials of the split-precision spherical kernel
(csrc/legendre.cuh), compiled for the host, against exact rational values."""
import ctypes as C
import os
import random
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hack_wein2k_b200", "csrc")
LMAX = 12
SRC = """#include "legendre.cuh"
extern "C" void leg(int l, int n, const double* x, double* w) {
  for (int i = 0; i < n; i++) {
    const double a[1] = {x[i]};
    double b[1];
    switch (l) {
%s
    }
    w[i] = b[0];
  }
}
""" % "\n".join(f"      case {l}: leg_poly<{l}>(a, b); break;" for l in range(LMAX + 1))


@pytest.fixture(scope="module")
def leg(tmp_path_factory):
    d = tmp_path_factory.mktemp("leg")
    (d / "leg.cpp").write_text(SRC)
    so = str(d / "leg.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-I", CSRC,
                           f"-DSPH_LMAX={LMAX + 1}", "-D__host__=", "-D__device__=", "-D__forceinline__=inline",
                           "-o", so, str(d / "leg.cpp")])
    lib = C.CDLL(so)
    lib.leg.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_void_p]

    def call(l, x):
        w = np.empty_like(x)
        lib.leg(l, x.size, x.ctypes.data, w.ctypes.data)
        return w

    return call


def _exact(l, x):
    p0, p1 = Fraction(1), x
    if l == 0:
        return p0
    for k in range(2, l + 1):
        p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
    return (2 * l + 1) * p1


@pytest.mark.parametrize("l", range(LMAX + 1))
def test_weights_are_exact_to_one_rounding_of_x(leg, l):
    """(2l+1) P_l(x) within (2l+1) l (l+1) / 2 eps, eps = 2^-53: the change at
    x = 1, where it is steepest, for an x off by one rounding (and one eps for
    l = 0)."""
    rng = random.Random(l)
    x = ([rng.uniform(-1.0, 1.0) for _ in range(400)] + [rng.uniform(0.95, 1.0) for _ in range(400)]
         + [1.0 - rng.uniform(0.0, 1e-6) for _ in range(50)] + [0.0, 1.0, -1.0, 0.5 ** 0.5])
    x = np.array(x)
    w = leg(l, x)
    tol = 2.0 ** -53 * max(1.0, (2 * l + 1) * l * (l + 1) / 2)
    err = max(abs(float(Fraction(float(a)) - _exact(l, Fraction(float(b))))) for a, b in zip(w, x))
    assert err <= tol, (l, err, tol)
