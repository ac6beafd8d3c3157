"""GPU: the memory of one call's arrays, which a context keeps between calls.

Threads that smooth different fields through one context, each on a stream of
its own, get the fields that one thread gets (bit-identical: an array handed
from one stream to another before its user was done would show); after a call
whose array is larger than what a context may keep (256 MiB) no more than that
is held, and closing the context gives the rest back (32 MiB of slack for the
driver's own needs)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _smooth(f, ctx, stream=None):
    from surfattpp_b200 import postproc
    ny, nz = f.shape[1:]
    return postproc.pde_smooth(f, 24.0 + 0.05 * np.arange(ny), 2.0 * np.arange(nz), 0.05, 0.05,
                               2.0, 0.12, 4.0, ctx=ctx, stream=stream)[0]


@pytest.mark.parametrize("shapes", [[(31, 33, 15)] * 4, [(90, 80, 30), (41, 41, 30), (61, 70, 33),
                                                       (120, 100, 20)]])
def test_threads_and_streams(gpu, shapes):
    import torch
    from surfattpp_b200 import _capi
    ctx = _capi.Context(0)
    gen = torch.Generator(device="cuda:0").manual_seed(3)
    fields = [torch.randn(s, generator=gen, device="cuda:0", dtype=torch.float64) for s in shapes]
    ref = [_smooth(f.clone(), ctx) for f in fields]
    got = [[] for _ in fields]
    torch.cuda.synchronize()

    def run(i):
        st = torch.cuda.Stream()
        for _ in range(10):
            with torch.cuda.stream(st):
                f = fields[i].clone()
                _smooth(f, ctx, st.cuda_stream)
            got[i].append(f)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(fields))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for r, g in zip(ref, got):
        assert len(g) == 10 and all(torch.equal(r, x) for x in g)
    ctx.close()


def test_bounded_and_given_back(gpu):
    import torch
    from surfattpp_b200 import _capi
    f = torch.zeros(601, 601, 110, device="cuda:0", dtype=torch.float64)   # 303 MiB
    torch.cuda.synchronize()
    start = torch.cuda.mem_get_info()[0]
    ctx = _capi.Context(0)
    for _ in range(2):
        _smooth(f, ctx)
        _smooth(f[:300].clone(), ctx)
    torch.cuda.empty_cache()
    assert start - torch.cuda.mem_get_info()[0] <= (256 + 32) * MIB
    ctx.close()
    torch.cuda.empty_cache()
    assert start - torch.cuda.mem_get_info()[0] <= 32 * MIB
