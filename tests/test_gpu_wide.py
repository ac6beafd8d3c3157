"""Few events: a block per event (several warps a solve) against the oracle
and against a warp per event.  Grids with rows at the edges of warps and of
the largest blocks (384 rows FP64, 512 FP32), wide and tall.

FP64: receiver times, iteration counts, and adj_s and chi with event-order
sums, bit for bit the oracle's.  FP32: the same events repeated until every
warp has its own give the same bits for times and iteration counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(40, 31), (33, 32), (35, 33), (90, 64), (21, 65), (37, 129), (12, 385), (15, 513)]


def _events(nx, ny, ne, topo):
    g = np.random.default_rng(nx * 1000 + ny)
    xx, yy = 102.0 + 0.02 * np.arange(nx), 24.0 + 0.02 * np.arange(ny)
    shp = (2, ny, nx)
    svel = 3.2 * (1.0 + 0.1 * g.uniform(-1, 1, shp))
    if topo:
        fx, fy = g.normal(0, 0.3, shp), g.normal(0, 0.3, shp)
        den = 1 + fx ** 2 + fy ** 2
        med = [(1 + fy ** 2) / den, -fx * fy / den, (1 + fx ** 2) / den]
    else:
        med = [np.ones(shp), np.full(shp, -0.0), np.ones(shp)]
    nr = 6
    ev = dict(evlo=g.uniform(xx[1], xx[-2], ne), evla=g.uniform(yy[1], yy[-2], ne),
              iper=np.arange(ne, dtype=np.int32) % 2, rec_ptr=nr * np.arange(ne + 1, dtype=np.int32),
              rec_idx=g.integers(0, 9, ne * nr).astype(np.int32),
              stlo=g.uniform(xx[0], xx[-1], 9), stla=g.uniform(yy[0], yy[-1], 9),
              tt_obs=g.uniform(5, 60, ne * nr), weight=g.uniform(0.5, 2, ne * nr))
    return xx, yy, svel, med, ev


def _run(xx, yy, svel, med, ev, precision, determ=False):
    import torch
    from surfattpp_b200 import preproc
    plan = preproc.ForwardAdjointPlan(xx, yy, 2, ev["evlo"], ev["evla"], ev["iper"], ev["rec_ptr"],
                                      ev["rec_idx"], ev["stlo"], ev["stla"], precision=precision)
    if determ:
        plan.set_deterministic()
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda:0")   # noqa: E731
    m = [None] * 3 if med is None else [t(v) for v in med]
    out = plan.run(t(svel), t(ev["tt_obs"]), t(ev["weight"]), True, *m)
    torch.cuda.synchronize()
    return {k: v.cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("topo", [False, True])
def test_fp64_matches_oracle_bits(gpu, orc, nx, ny, topo):
    xx, yy, svel, med, ev = _events(nx, ny, 5, topo)
    got = _run(xx, yy, svel, med if topo else None, ev, "fp64", determ=True)
    ref = orc.forward_for_events(xx, yy, svel, *med, ev, math="cr")
    assert np.array_equal(got["fwd_iters"], ref["fwd_iters"])
    assert np.array_equal(got["adj_iters"], ref["adj_iters"])
    assert np.array_equal(got["syn"], ref["syn"])
    assert np.array_equal(got["adj_s"], ref["adj_s"])
    assert got["chi"][0] == ref["chi"]


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("topo", [False, True])
def test_fp32_block_equals_warp(gpu, nx, ny, topo):
    ne, rep = 4, 600      # 2400 events: a warp each
    xx, yy, svel, med, ev = _events(nx, ny, ne, topo)
    med = med if topo else None
    few = _run(xx, yy, svel, med, ev, "fp32")
    many = dict(ev, **{k: np.tile(ev[k], rep) for k in ("evlo", "evla", "iper", "rec_idx", "tt_obs",
                                                        "weight")})
    many["rec_ptr"] = np.arange(ne * rep + 1, dtype=np.int32) * 6
    all_ = _run(xx, yy, svel, med, many, "fp32")
    for k in ("syn", "fwd_iters", "adj_iters"):
        assert np.array_equal(np.tile(few[k], rep), all_[k])
    assert few["status"].max() == 0
    assert np.allclose(all_["adj_s"], rep * few["adj_s"], rtol=1e-12, atol=1e-12 * np.abs(all_["adj_s"]).max())
