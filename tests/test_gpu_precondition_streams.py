"""sa_kernel_precondition returns before it has run; calls on different streams
of one context overlap and must not share their maxima's partial results.
Densities of very different maxima, a size of many blocks; every result has
to be the one that the call gives alone, bit for bit.  Under capture a call
replays on new data, and one beside a capture leaves it alone."""
import pytest

pytestmark = pytest.mark.gpu


def _inputs(n, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    den = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 10.0 ** (3 * seed)
    return den, torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


@pytest.mark.parametrize("n", [1000, 3_000_017])
def test_streams_overlap(gpu, n):
    import torch
    from surfattpp_b200 import postproc
    data = [_inputs(n, k) for k in range(3)]
    alone = []
    for den, ker in data:
        k = ker.clone()
        postproc.kernel_precondition(den, k)
        torch.cuda.synchronize()
        alone.append(k)
    streams = [torch.cuda.Stream() for _ in data]
    for _ in range(20):
        got = [ker.clone() for _, ker in data]
        torch.cuda.synchronize()
        for s, k, (den, _) in zip(streams, got, data):
            postproc.kernel_precondition(den, k, stream=s.cuda_stream)
        torch.cuda.synchronize()
        for k, a in zip(got, alone):
            assert torch.equal(k, a)


def test_capture(gpu):
    import torch
    from surfattpp_b200 import postproc
    den, ker = _inputs(100_003, 1)
    k = ker.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        postproc.kernel_precondition(den, k, stream=torch.cuda.current_stream().cuda_stream)
    for seed in (2, 3):
        d2, k2 = _inputs(100_003, seed)
        want = k2.clone()
        postproc.kernel_precondition(d2, want)
        torch.cuda.synchronize()
        den.copy_(d2)
        k.copy_(k2)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(k, want)


def test_beside_a_capture(gpu):
    import torch
    from surfattpp_b200 import postproc
    den, ker = _inputs(100_003, 1)
    want, got = ker.clone(), ker.clone()
    postproc.kernel_precondition(den, want)
    k, other = ker.clone(), torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        postproc.kernel_precondition(den, k, stream=torch.cuda.current_stream().cuda_stream)
        postproc.kernel_precondition(den, got, stream=other.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(k, want) and torch.equal(got, want)
