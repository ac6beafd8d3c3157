"""The FP64 forward update, which evaluates only the stencils that can lower a
cell, against the oracle, which evaluates them all: travel times bit for bit
and the same iteration counts where the decision is closest -- cells next to
the source (on a node, on a grid line, in a cell's middle, on the edge), rays
along the axes and the diagonals of a homogeneous medium, strong cross terms,
uneven spacing, rough slowness and the smallest and slender grids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(nx, ny, step, stretch, src, medium):
    g = np.random.default_rng(nx * 1000 + ny)
    xx, yy = 102.0 + step * np.arange(nx), 24.0 + step * stretch * np.arange(ny)
    x0 = {"node": xx[nx // 2], "line": xx[nx // 2], "middle": xx[nx // 2 - 1] + 0.5 * step,
          "edge": xx[0]}[src]
    y0 = {"node": yy[ny // 2], "line": yy[ny // 2 - 1] + 0.31 * (yy[1] - yy[0]),
          "middle": yy[ny // 2 - 1] + 0.5 * (yy[1] - yy[0]), "edge": yy[-1]}[src]
    one = np.ones((ny, nx))
    if medium == "homogeneous":
        return xx, yy, one, one.copy(), 0.0 * one, one / 3.0, x0, y0
    rough = 1.0 / (3.2 * (1.0 + 0.4 * g.uniform(-1, 1, one.shape)))
    if medium == "rough":
        return xx, yy, one, one.copy(), 0.0 * one, rough, x0, y0
    fx, fy = g.normal(0, 1.5, one.shape), g.normal(0, 1.5, one.shape)   # steep slopes
    den = 1.0 + fx ** 2 + fy ** 2
    return xx, yy, (1 + fy ** 2) / den, (1 + fx ** 2) / den, fx * fy / den, rough, x0, y0


@pytest.mark.parametrize("nx,ny,step,stretch", [(3, 3, 0.05, 1.0), (4, 70, 0.01, 1.0),
                                                (33, 32, 0.002, 1.0), (65, 31, 0.05, 2.3),
                                                (97, 64, 0.3, 0.4)])
@pytest.mark.parametrize("src", ["node", "line", "middle", "edge"])
@pytest.mark.parametrize("medium", ["homogeneous", "rough", "steep"])
def test_solve_matches_oracle_bits(gpu, orc, nx, ny, step, stretch, src, medium):
    from surfattpp_b200 import eikonal
    case = _case(nx, ny, step, stretch, src, medium)
    T, it = eikonal.FSM_UW_PS_lonlat_2d(*case, return_iters=True)
    ref, rit = orc.eik_fwd(*case)
    assert it == rit
    assert np.array_equal(T, ref)


@pytest.mark.parametrize("src", ["node", "line", "middle", "edge"])
@pytest.mark.parametrize("medium", ["homogeneous", "rough"])
def test_isotropic_batch_matches_oracle_bits(gpu, orc, src, medium):
    from surfattpp_b200 import preproc
    xx, yy, one, _, zero, fun, x0, y0 = _case(47, 38, 0.02, 1.3, src, medium)
    g = np.random.default_rng(5)
    n = 40
    ev = dict(evlo=np.array([x0]), evla=np.array([y0]), iper=np.zeros(1, np.int32),
              rec_ptr=np.array([0, n], np.int32), rec_idx=np.arange(n, dtype=np.int32),
              stlo=g.uniform(xx[0], xx[-1], n), stla=g.uniform(yy[0], yy[-1], n),
              tt_obs=np.zeros(n), weight=np.ones(n))
    svel = (1.0 / fun)[None]
    out = preproc.forward_for_event(xx, yy, svel, ev)
    ref = orc.forward_for_events(xx, yy, svel, one[None], -zero[None], one[None], ev)
    assert np.array_equal(out["fwd_iters"], ref["fwd_iters"])
    assert np.array_equal(out["syn"], ref["syn"])
