"""fwdsurf by a thread per column and by groups of 32, 16 and 8 lanes (chosen
by the number of columns): velocities and statuses bit-identical to the
oracle with the same correctly rounded functions, for Rayleigh and Love phase
and group velocities.  The columns repeat a set with a low-velocity zone, a
soft top, a water layer, layers of uneven thickness and two or many layers,
so that marches end in every way (a root, below the start, no root)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _columns(nz, n=61):
    g = np.random.default_rng(nz)
    z = np.cumsum(np.r_[0.0, 1.0 + 2.0 * g.random(nz - 1)])
    vs = np.empty((n, nz))
    for i in range(n):
        v0, v1 = (0.6, 3.5) if i % 7 == 3 else (2.8, 4.6)
        vs[i] = (v0 + (v1 - v0) * z / z[-1]) * (1 + 0.15 * np.clip(g.standard_normal(nz), -1, 1))
        if i % 9 == 4:
            vs[i, nz // 3:nz // 2] *= 0.7
        if i % 20 == 11:
            vs[i, 0] = 0.0
    return z, vs


# columns: a few, the ends of the 32-, 16- and 8-lane ranges on 148 SMs (with a
# last block that is not full), and a thread per column
@pytest.mark.parametrize("ncol", [1, 7, 2367, 2369, 4737, 35521])
@pytest.mark.parametrize("iwave,igr,nz", [(2, 0, 30), (2, 1, 2), (1, 0, 63), (1, 1, 17)])
def test_columns_match_oracle(gpu, orc, ncol, iwave, igr, nz):
    import torch
    from surfattpp_b200 import surfker
    z, vs = _columns(nz)
    p = np.geomspace(2.0, 40.0, 5)
    ref, st = orc.fwdsurf(z, vs[:, None, :], p, iwave=iwave, igr=igr, nthreads=8, math="cr")
    k = np.arange(ncol) % vs.shape[0]
    dev = torch.as_tensor(np.ascontiguousarray(vs[k][:, None, :]), device="cuda:0")
    got, status = surfker.fwdsurf(z, dev, p, iwave=iwave, igr=igr, check=False)
    assert np.array_equal(status.cpu().numpy()[0], st[0][k])
    assert np.array_equal(got.cpu().numpy()[:, 0, :], ref[:, 0, :][:, k], equal_nan=True)
