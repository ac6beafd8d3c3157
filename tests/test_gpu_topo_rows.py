"""Topography smoothing with a row's weights shared between its cells (evenly
spaced longitudes) and with a weight per point (uneven ones), against the
oracle: media within 1e-12 and dip angles within 1e-9 degrees, the bars of
the per-point form.  Windows of one point, a few, wider than the grid; grids
narrower than a warp, ragged, and wider than a block; spacing rounded to
FP32 and stretched, which have to take the per-point form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(3, 3), (31, 12), (70, 33), (263, 9)])
@pytest.mark.parametrize("spacing", ["even", "float32", "stretched"])
def test_media_match_oracle(gpu, orc, nx, ny, spacing):
    import torch
    from surfattpp_b200 import surfgrid
    g = np.random.default_rng(nx + ny)
    x, y = 102.0 + 0.01 * np.arange(nx), 24.0 + 0.013 * np.arange(ny)
    if spacing == "float32":
        x = x.astype(np.float32).astype(np.float64)
    elif spacing == "stretched":
        x = 102.0 + 0.01 * np.arange(nx) * (1 + 0.001 * np.arange(nx))
    z = g.uniform(0, 4, (ny, nx))
    sig = np.array([0.002, 0.0123, 0.06, 1.1])
    zt = torch.as_tensor(z, device="cuda:0")
    got = [v.cpu().numpy() for v in surfgrid.build_media_with_topo(x, y, zt, sig)]
    ref = orc.topo_media(x, y, z, sig)
    for a, b in zip(got[:3], ref[:3]):
        assert np.abs(a - b).max() <= 1e-12
    assert np.abs(got[3] - ref[3]).max() <= 1e-9
