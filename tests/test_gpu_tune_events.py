"""What the launch autotuner found for many events on a grid is not handed to
plans of few events, which a block per event serves, nor the other way round;
plans of as many events, and of more in the same form, take it in proportion
to their slots."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(w, ev, ne, ctx):
    from surfattpp_b200 import preproc
    sel = np.arange(ne) % ev["iper"].size
    ptr = [0]
    idx = []
    for e in sel:
        r = ev["rec_idx"][ev["rec_ptr"][e]:ev["rec_ptr"][e + 1]]
        idx.append(r)
        ptr.append(ptr[-1] + r.size)
    pairs = np.concatenate([np.arange(ev["rec_ptr"][e], ev["rec_ptr"][e + 1]) for e in sel])
    p = preproc.ForwardAdjointPlan(w.xx_deg, w.yy_deg, w.nper, ev["evlo"][sel], ev["evla"][sel],
                                   ev["iper"][sel], np.array(ptr), np.concatenate(idx),
                                   ev["stlo"], ev["stla"], precision="fp32", ctx=ctx)
    return p, pairs


@pytest.mark.parametrize("tuned,other", [(3000, 40), (40, 3000)])
def test_tuned_choice_stays_with_its_form(gpu, tuned, other):
    import torch
    from surfattpp_b200 import _capi
    from surfattpp_b200 import workloads as W
    w = W.config3(nsta=25, nper=4, n=81)
    ev = w.events()
    dev = torch.device("cuda", 0)
    sv = torch.full((w.nper, w.ny, w.nx), 3.0, dtype=torch.float64, device=dev)
    # several contexts: the fastest candidate varies
    for _ in range(3):
        ctx = _capi.Context(0)
        p, pairs = _plan(w, ev, tuned, ctx)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        got = p.autotune(sv, t(ev["tt_obs"][pairs]), t(ev["weight"][pairs]))
        q, _ = _plan(w, ev, other, ctx)
        assert (q.tune()["variant"], q.tune()["active_slots"]) == (0, q.tune()["nslots"])
        r, _ = _plan(w, ev, tuned, ctx)
        assert r.tune() == p.tune()
        assert (r.tune()["variant"], r.tune()["active_slots"]) == (got["variant"],
                                                                  got["active_slots"])
        for x in (p, q, r):
            x.close()
