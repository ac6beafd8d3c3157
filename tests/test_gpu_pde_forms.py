"""GPU parity: the PDE smoothing's forms (all steps in one cluster launch for a
small field, two steps per pass for a large one) against the oracle.

Sizes at the edges of the forms' tiles: fewer rows than a row group, the last
row first or last in a group, blocks of the cluster without a group, a field
just within and just beyond the cluster's threads; depths just within and
beyond one tile, rows and planes that leave short last tiles, odd and even
step counts (the first pass reads the boundary as given, later ones the
clamped interior).

Bar: bit-identical (every form evaluates each cell's update with the same
operations in the same order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER = [(3, 3, 3), (4, 5, 3), (5, 3, 4), (3, 41, 6), (18, 6, 3), (19, 7, 11), (31, 33, 15),
           (41, 41, 30), (35, 30, 50), (5, 8, 66), (34, 32, 34), (34, 32, 35), (66, 28, 36)]
PASS = [(262, 40, 202), (700, 61, 50), (121, 270, 65), (131, 254, 64), (1203, 110, 16),
        (34, 902, 69), (34, 903, 70), (300, 301, 24)]


def _check(orc, shape, steps):
    import torch
    from surfattpp_b200 import postproc
    nx, ny, nz = shape
    d, dz = 0.05, 2.0
    y, z = 24.0 + 0.01 * np.arange(ny), dz * np.arange(nz)
    # the horizontal width that takes `steps` steps
    cm = min(d * d * np.cos(np.radians(y[-1])) ** 2, d * d) / 6.0
    sh = np.sqrt(2.0 * cm * (steps - 0.5))
    f = np.random.default_rng([*shape, steps]).standard_normal(shape)
    ref, ns = orc.pde_smooth(f, d, d, dz, y, z, sh, 0.5)
    assert ns == steps
    t = torch.as_tensor(f, device="cuda:0").contiguous()
    out, got = postproc.pde_smooth(t, y, z, d, d, dz, sh, 0.5)
    torch.cuda.synchronize()
    assert got == steps and np.array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("steps", [1, 2, 7])
@pytest.mark.parametrize("shape", CLUSTER)
def test_small(gpu, orc, shape, steps):
    _check(orc, shape, steps)


@pytest.mark.parametrize("steps", [1, 2, 3, 6])
@pytest.mark.parametrize("shape", PASS)
def test_large(gpu, orc, shape, steps):
    _check(orc, shape, steps)
