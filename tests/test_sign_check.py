"""The dispersion search's march takes signs from approximate secular functions
where they stand above 1e-6 of the normalised vector (kSignSure).  Host build:
where they are trusted they lie within a tenth of that of the exact ones, in
the form with a thread per column and in that with tables, for any trial
velocity, those next to a layer's or the half-space's among them, for layers of
many wavelengths, and for periods beyond dltar4's smallest frequency."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "surfattpp_b200", "csrc")
OUT = os.path.join(HERE, "_build", "libsign_check.so")
BOUND = 1e-7


@pytest.fixture(scope="module")
def lib():
    src = os.path.join(HERE, "sign_check.cpp")
    deps = [src] + [os.path.join(CSRC, f) for f in ("surfker_search.cuh", "surfker_dev.cuh",
                                                    "crmath.cuh", "crmath_tables.h")]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                        "-I", CSRC, "-I", "/usr/local/cuda/include", "-o", OUT, src], check=True)
    L = C.CDLL(OUT)
    L.sign_check.restype = C.c_double
    L.sign_check.argtypes = [C.c_int] * 3 + [C.c_double] * 4 + [C.c_long, C.c_ulong,
                                                               C.POINTER(C.c_long)]
    return L


def _worst(lib, love, tables, where, periods, thickness, n=20_000):
    untrusted = C.c_long()
    w = lib.sign_check(love, tables, where, *periods, *thickness, n, 5 + where, C.byref(untrusted))
    return w, untrusted.value / n


@pytest.mark.parametrize("love", [0, 1])
@pytest.mark.parametrize("tables", [0, 1])
@pytest.mark.parametrize("periods", [(1.0, 60.0), (100.0, 6e4), (6.3e4, 1e6)])
def test_any_velocity(lib, love, tables, periods):
    worst, untrusted = _worst(lib, love, tables, 0, periods, (0.3, 5.0))
    assert worst <= BOUND and untrusted < 0.01


@pytest.mark.parametrize("love", [0, 1])
@pytest.mark.parametrize("tables", [0, 1])
@pytest.mark.parametrize("where", [1, 2, 3])
def test_next_to_a_velocity(lib, love, tables, where):
    worst, untrusted = _worst(lib, love, tables, where, (1.0, 60.0), (0.3, 5.0))
    assert worst <= BOUND and untrusted < 0.02


@pytest.mark.parametrize("love", [0, 1])
@pytest.mark.parametrize("tables", [0, 1])
@pytest.mark.parametrize("where", [0, 2])
@pytest.mark.parametrize("periods", [(0.05, 1.0), (0.002, 0.05), (1e-4, 0.002)])
def test_many_wavelengths(lib, love, tables, where, periods):
    """Not trusted, or accurate."""
    worst, _ = _worst(lib, love, tables, where, periods, (10.0, 60.0))
    assert worst <= BOUND
