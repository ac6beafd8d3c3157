"""The short evaluations of exp, log and sincos (crmath.cuh), taken where
their rounding test passes, return the full evaluation's bits; nearly every
argument takes them.  Arguments at the edges: the ends of the accepted range,
table-interval boundaries, zeros and quarter turns, and random ones between."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "surfattpp_b200", "csrc")
OUT = os.path.join(HERE, "_build", "libcrmath_short_check.so")


@pytest.fixture(scope="module")
def lib():
    src = os.path.join(HERE, "crmath_short_check.cpp")
    deps = [src, os.path.join(CSRC, "crmath.cuh"), os.path.join(CSRC, "crmath_tables.h")]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                        "-I", CSRC, "-o", OUT, src], check=True)
    L = C.CDLL(OUT)
    L.cr_short_check.argtypes = [C.c_int, C.c_void_p, C.c_long, C.POINTER(C.c_long)]
    L.cr_short_check.restype = C.c_long
    return L


def _args(f, n=100_000):
    g = np.random.default_rng(7 + f)
    if f == 0:
        k = np.arange(-4096, 4096) * (np.log(2.0) / 4096) * 0.5   # interval centres and edges
        return np.concatenate([g.uniform(-708, 708, n), g.uniform(-60, 0, n), k,
                               -np.exp(g.uniform(-40, 3, n)), [708.0, -708.0, 0.0, -0.0]])
    if f == 1:
        e = 1.0 + np.arange(128) / 128.0                            # table boundaries
        return np.concatenate([np.exp(g.uniform(-690, 690, n)), g.uniform(0.5, 2, n), e,
                               np.nextafter(e, 0), e / 2, 1 + np.exp(g.uniform(-35, -1, n)),
                               1 - 0.9 * np.exp(g.uniform(-35, -1, n)), [2.0 ** -1000, 2.0 ** 1000]])
    q = np.arange(-2000, 2000) * (np.pi / 2)
    return np.concatenate([g.uniform(-50, 50, n), g.uniform(-3215, 3215, n), q * (1 + 1e-7),
                           q + 1e-5, np.arange(202) / 256 + 1 / 512,
                           np.exp(g.uniform(-13, 1, n)), -np.exp(g.uniform(-13, 1, n))])


@pytest.mark.parametrize("f", [0, 1, 2])
def test_short_equals_full(lib, f):
    x = np.ascontiguousarray(_args(f))
    taken = C.c_long()
    assert lib.cr_short_check(f, x.ctypes.data, x.size, C.byref(taken)) == 0
    assert taken.value > 0.95 * x.size
