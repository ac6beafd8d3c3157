"""sa_topo_media at the ends of what it accepts: windows wider than any grid,
coordinates and topography that are not finite, more periods than a launch's
grid holds, tall grids.  Bars: media within 1e-12 and dip angles within 1e-9 degrees of
the oracle, the bars of the ordinary cases; non-finite values in the same
cells as the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _media(x, y, z, sig):
    import torch
    from surfattpp_b200 import surfgrid
    zt = torch.as_tensor(z, device="cuda:0")
    return [v.cpu().numpy() for v in surfgrid.build_media_with_topo(x, y, zt, np.asarray(sig))]


def _match(got, ref):
    for a, b, tol in zip(got, ref, (1e-12, 1e-12, 1e-12, 1e-9)):
        f = np.isfinite(b)
        assert np.array_equal(np.isfinite(a), f)
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.abs(a[f] - b[f]).max() <= tol


def _grid(nx, ny, seed):
    g = np.random.default_rng(seed)
    return 102.0 + 0.01 * np.arange(nx), 24.0 + 0.013 * np.arange(ny), g.uniform(0, 4, (ny, nx))


@pytest.mark.parametrize("wide", [1e8, 1e30, np.inf])
def test_window_beyond_integers(gpu, orc, wide):
    """Beside a period whose window in grid points exceeds an integer, the
    others come out as ever."""
    x, y, z = _grid(70, 33, 1)
    got = _media(x, y, z, [0.0123, wide, 0.061])
    ref = orc.topo_media(x, y, z, np.array([0.0123, 0.061]))
    _match([a[::2] for a in got], ref)


@pytest.mark.parametrize("axis,bad", [("x", np.nan), ("x", np.inf), ("y", np.nan)])
def test_coordinate_not_finite(gpu, axis, bad):
    """A point at no position has no weight: cells away from it (and from the
    gradients that difference it) stay finite."""
    x, y, z = _grid(70, 33, 2)
    k = 20
    (x if axis == "x" else y)[k] = bad
    for a in _media(x, y, z, [0.061]):
        keep = np.delete(a, [k - 1, k, k + 1], axis=2 if axis == "x" else 1)
        assert np.isfinite(keep).all()


@pytest.mark.parametrize("bad", [[np.nan], [np.inf], [-np.inf], [np.inf, -np.inf]])
@pytest.mark.parametrize("nx,ny", [(31, 12), (70, 33), (263, 9)])
def test_topography_not_finite(gpu, orc, nx, ny, bad):
    """A non-finite cell reaches the cells whose window holds it, no others."""
    x, y, z = _grid(nx, ny, 3)
    for i, v in enumerate(bad):
        z[ny // 2, nx // 2 + 3 * i] = v
    z[0, nx - 1] = bad[0]
    sig = np.array([0.002, 0.0123, 0.031])
    _match(_media(x, y, z, sig), orc.topo_media(x, y, z, sig))


def test_more_periods_than_a_grid_holds(gpu, orc):
    x, y, z = _grid(3, 3, 4)
    sig = np.full(65540, 0.0123)
    sig[-1] = 0.031
    got = _media(x, y, z, sig)
    _match([a[-2:] for a in got], orc.topo_media(x, y, z, sig[-2:]))
    for a in got:
        assert np.array_equal(a[0], a[65535])


@pytest.mark.parametrize("nx,ny", [(5, 3072), (5, 3073), (131, 4001), (3, 14528)])
def test_tall_grids(gpu, orc, nx, ny):
    """More latitudes than the per-point form has shared memory for without
    asking for more."""
    x, y, z = _grid(nx, ny, 5)
    y = 24.0 + 0.0004 * np.arange(ny)
    z[ny // 2, nx // 2] = np.nan
    sig = np.array([0.011])
    _match(_media(x, y, z, sig), orc.topo_media(x, y, z, sig))
