"""The branch-free reciprocals, quotients and square roots of rounded.cuh
against CUDA's IEEE operations, bit for bit, on the device: random operands,
mantissas of ones and powers of two, quotients and roots next to a midpoint
of two doubles, exact squares and their neighbours.  A root that is not sure
(the caller then takes CUDA's) may be rare only where operands are random."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "surfattpp_b200", "csrc")
OUT = os.path.join(HERE, "_build", "librounded_check.so")


@pytest.fixture(scope="module")
def lib():
    from surfattpp_b200 import build
    src = os.path.join(HERE, "rounded_check.cu")
    deps = [src, os.path.join(CSRC, "rounded.cuh")]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "-fmad=false", "-shared",
                        "-Xcompiler", "-fPIC", "-I", CSRC, "-o", OUT, src], check=True)
    L = C.CDLL(OUT)
    L.rounded_check.argtypes = [C.c_int, C.c_long, C.c_ulong, C.POINTER(C.c_ulonglong)]
    return L


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
def test_rounds_as_ieee(gpu, lib, kind):
    n = 4_000_000
    bad = (C.c_ulonglong * 4)()
    assert lib.rounded_check(kind, n, 11 + kind, bad) == 0
    assert list(bad[:3]) == [0, 0, 0]
    if kind == 0:
        assert bad[3] <= 3
