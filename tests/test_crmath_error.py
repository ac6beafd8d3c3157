"""The short evaluations of exp, log and sincos (crmath.cuh) leave an error of
at most half of what their rounding test allows, against quad precision:
arguments at both ends and in the middle of every table interval, where the
series' remainders are largest, next to 1 and to multiples of pi/2, and random
ones over the accepted range."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "surfattpp_b200", "csrc")
OUT = os.path.join(HERE, "_build", "libcrmath_error_check.so")


@pytest.fixture(scope="module")
def lib():
    src = os.path.join(HERE, "crmath_error_check.cpp")
    deps = [src, os.path.join(CSRC, "crmath.cuh"), os.path.join(CSRC, "crmath_tables.h")]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run(["g++", "-O2", "-std=gnu++17", "-fPIC", "-shared", "-ffp-contract=off",
                        "-I", CSRC, "-o", OUT, src, "-lquadmath"], check=True)
    L = C.CDLL(OUT)
    L.cr_short_error.argtypes = [C.c_int, C.c_void_p, C.c_long, C.POINTER(C.c_double)]
    L.cr_short_error.restype = C.c_double
    return L


def _args(f, n=60_000):
    g = np.random.default_rng(17 + f)
    near = 1.0 + np.array([-1, 1]) * np.exp(g.uniform(-30, -5, n))[:, None]
    if f == 0:
        edge = (np.arange(-20_000, 20_000) + 0.5) * (np.log(2.0) / 4096)
        return np.concatenate([g.uniform(-708, 708, n), edge, edge * near[:40_000, 0],
                               -np.exp(g.uniform(-40, 4, n))])
    if f == 1:
        j = 1.0 + np.arange(129) / 128.0
        ends = np.concatenate([j[:-1, None] * (1 + np.exp(g.uniform(-30, -5, (128, 200)))),
                               j[1:, None] * (1 - np.exp(g.uniform(-30, -5, (128, 200))))])
        ends = np.concatenate([ends.ravel(), g.uniform(1, 1.02, n), g.uniform(0.98, 1, n)])
        return np.concatenate([ends, ends * 0.5, ends * 2.0, ends * 2.0 ** 40,
                               np.exp(g.uniform(-690, 690, n)), near.ravel()])
    q = np.arange(-2000, 2000) * (np.pi / 2)
    t = (np.arange(0, 202) + 0.5) / 256
    return np.concatenate([g.uniform(-50, 50, n), g.uniform(-3215, 3215, n), q + 2e-6, q - 1e-4,
                           (t[:, None] * near[:200].ravel()).ravel(),
                           np.exp(g.uniform(-13, 1, n))])


@pytest.mark.parametrize("f", [0, 1, 2])
def test_error_is_half_of_what_is_allowed(lib, f):
    x = np.ascontiguousarray(_args(f))
    at = C.c_double()
    share = lib.cr_short_error(f, x.ctypes.data, x.size, C.byref(at))
    assert share <= 0.5, at.value
