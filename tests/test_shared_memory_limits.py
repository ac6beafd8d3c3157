"""A kernel's limit on dynamic shared memory belongs to the device: one that is
set to the need of the call at hand can be lowered by another thread before
that call's launch.  Every place that sets it sets a constant."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "surfattpp_b200", "csrc")


def test_limits_are_constants():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        src = open(os.path.join(CSRC, name)).read()
        for arg in re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize\s*,\s*([^;]*?)\)+;?\n",
                              src):
            found += 1
            assert re.fullmatch(r"\w+", arg), (name, arg)
            assert re.search(r"constexpr int [^;]*\b%s =" % arg, src), (name, arg)
    assert found >= 4
