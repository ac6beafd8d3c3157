"""Kernels launched as programmatic dependents are resident while the launch
before them still writes.  `__restrict__` tells the compiler that an array
keeps its values for the kernel's lifetime (and lets it load a const one
through the read-only path, which the dependency does not cover), so only
arrays that no launch of such a chain writes may carry it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "surfattpp_b200", "csrc")
# kernel -> the arrays that its chain of launches only reads
ONLY_READ = {"pde_step_kernel32": {"rowX", "rowY", "depE"}, "lbfgs_pass_kernel": {"x", "d"}}


def test_changing_arrays_are_unqualified():
    seen = set()
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        src = open(os.path.join(CSRC, name)).read()
        for kernel in re.split(r"__global__", src)[1:]:
            if "cudaGridDependencySynchronize()" not in kernel.split("\n}\n")[0]:
                continue
            kernel = re.sub(r"__launch_bounds__\([^)]*\)", "", kernel)
            fn, args = re.search(r"(\w+)\s*\(([^)]*)\)\s*\{", kernel).groups()
            seen.add(fn)
            fixed = {a.split()[-1].lstrip("*") for a in args.split(",") if "__restrict__" in a}
            assert fixed <= ONLY_READ[fn], (name, fn, fixed - ONLY_READ[fn])
    assert seen == set(ONLY_READ)
