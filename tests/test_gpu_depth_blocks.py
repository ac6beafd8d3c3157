"""GPU: the depth kernels in blocks of equal size, whatever the number of
(column, period) items: a single item, counts around a warp, around one full
wave (148 blocks of 640 threads) and beyond it; the group kernels' three
phase-velocity runs in one launch of each form (32, 16, 8 lanes and a thread
per column).

The columns repeat a few columns in an order that puts each beside others, and
every copy's kernels must be those of the column's first copy in the smallest
launch (those of other tests are compared with the oracle), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Z = 3.0 * np.arange(9)
WAVE = 148 * 640


def _columns():
    rng = np.random.default_rng(4)
    base = np.linspace(2.9, 4.4, Z.size)
    return base * (1.0 + 0.03 * rng.standard_normal((7, Z.size)).cumsum(1) / 3.0)


@pytest.mark.parametrize("kind", ["phase", "group", "love"])
@pytest.mark.parametrize("nx,ny,nper", [(1, 1, 1), (1, 31, 1), (3, 11, 1), (149, 1, 2),
                                        (33, 31, 2), (60, 61, 2),
                                        (320, 148, 2), (320, 74, 4), (57, 1662, 1),
                                        (500, 97, 2), (480, 148, 4)])
def test_equal_blocks(gpu, orc, kind, nx, ny, nper):
    import torch
    from surfattpp_b200 import surfker
    cols = _columns()
    T = np.array([6.0, 9.0, 14.0, 22.0])[:nper]

    def run(vs):
        t = torch.as_tensor(np.ascontiguousarray(vs), device="cuda:0")
        if kind == "group":
            r = surfker.depthkernel_group(Z, t, T)
        elif kind == "love":
            r = surfker.depthkernel_love(Z, t, T, 1)
        else:
            r = surfker.depthkernel_hti(Z, t, T, surfker.fwdsurf(Z, t, T)[0])
        return [x.cpu().numpy() for x in r]

    one = run(cols[:, None, :])
    which = (np.arange(nx * ny) * 5 % 7).reshape(nx, ny)
    for got, ref in zip(run(cols[which]), one):
        assert np.array_equal(got, ref[:, 0][which])
