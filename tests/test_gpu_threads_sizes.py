"""Calls of different sizes from several threads at once: a kernel's limit on
dynamic shared memory belongs to the device, not to the call, so that of one
call must not fail another's launch.  Each thread has its own context and
stream; three repeat a small size as long as one repeats a large one; every
call has to succeed, with the first one's bits."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _smooth(shape):
    import torch
    from surfattpp_b200 import postproc
    nx, ny, nz = shape
    f0 = torch.as_tensor(np.random.default_rng(nx).standard_normal(shape), device="cuda:0")
    y, z = 24.0 + 0.1 * np.arange(ny), 2.0 * np.arange(nz)

    def call(ctx, st):
        f = f0.clone()
        postproc.pde_smooth(f, y, z, 0.1, 0.1, 2.0, 0.05, 0.5, ctx=ctx, stream=st)
        return f
    return call


def _dispersion(nx, nz):
    import torch
    from surfattpp_b200 import surfker
    z = np.linspace(0.0, 60.0, nz)
    vs = torch.as_tensor(np.broadcast_to(2.8 + 0.03 * z, (nx, 70, nz)).copy(), device="cuda:0")

    def call(ctx, st):
        return surfker.fwdsurf(z, vs, np.array([8.0]), ctx=ctx, stream=st)[0]
    return call


def _topo(nx, sigma):
    import torch
    from surfattpp_b200 import surfgrid
    x, y = 102.0 + 0.01 * np.arange(nx), 24.0 + 0.01 * np.arange(9)
    zt = torch.as_tensor(np.random.default_rng(nx).uniform(0, 4, (9, nx)), device="cuda:0")

    def call(ctx, st):
        return surfgrid.build_media_with_topo(x, y, zt, np.array([sigma]), ctx=ctx, stream=st)[0]
    return call


@pytest.mark.parametrize("kind,n", [("cluster", 4000), ("passes", 1000), ("dispersion", 1500),
                                    ("topography", 4000)])
def test_sizes_do_not_meet(gpu, kind, n):
    import torch
    from surfattpp_b200 import _capi
    small, large = {"cluster": (_smooth((10, 9, 8)), _smooth((41, 41, 30))),
                    "passes": (_smooth((700, 90, 34)), _smooth((200, 180, 60))),
                    "dispersion": (_dispersion(70, 4), _dispersion(70, 63)),
                    "topography": (_topo(12, 0.004), _topo(600, 1.0))}[kind]
    errors, done = [], threading.Event()

    def work(call, count):
        try:
            torch.cuda.set_device(0)
            ctx, s = _capi.Context(0), torch.cuda.Stream()
            with torch.cuda.stream(s):
                first = got = call(ctx, s.cuda_stream)
                i = 0
                while i < count and not done.is_set():
                    got = call(ctx, s.cuda_stream)
                    i += 1
                assert torch.equal(got, first)
        except BaseException as e:
            errors.append(e)
        if count < 10**9:
            done.set()
    threads = [threading.Thread(target=work, args=a)
               for a in [(large, n)] + 3 * [(small, 10**9)]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
