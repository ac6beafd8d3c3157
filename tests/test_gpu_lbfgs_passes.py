"""GPU parity: the L-BFGS history kept as pairs that are formed when an iterate
is stored, and the recursion's coefficients kept on the device, against the
oracle's two-loop recursion from the stored iterates alone.

Sizes around the reductions' blocks (256 threads, 1184 blocks); histories that
were stored anew, out of order, with gaps, or with a curvature s.y <= 0.

Bar: 1e-11 of the direction's maximum, as for the other L-BFGS tests (the log
of the model differs from the C library's by at most an ulp)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = 256 * 1184
# (iterates in the order they are stored, a repeated one with new values;
#  iterate asked for)
ORDERS = {
    "one": ([0], 0),
    "pair": ([0, 1], 1),
    "reversed": ([3, 2, 1, 0], 3),
    "last-anew": ([0, 1, 2, 2], 2),
    "middle-anew": ([0, 1, 2, 3, 1], 3),
    "earlier": ([0, 1, 2, 3, 4], 2),
    "far-apart": ([0, 1, 10, 11], 1),
    "wrapped": (list(range(13)), 12),
    "back": ([4, 5, 6, 7, 8, 9, 3, 4], 8),
}


def _t(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda:0")


@pytest.mark.parametrize("n", [1, 2, 255, 257, GRID - 1, GRID, GRID + 1])
@pytest.mark.parametrize("order", list(ORDERS))
def test_direction(gpu, orc, order, n):
    from surfattpp_b200 import optimize
    stored, ask = ORDERS[order]
    rng = np.random.default_rng([n, len(order)])
    lb = optimize.LBFGS(n)
    have = {}
    for k in stored:
        m = np.exp(rng.normal(1.2, 0.05, n))
        g = rng.normal(size=n)
        if k - 1 in have:   # y along s, against it every third time
            c = 2.0 if k % 3 else -2.0
            g = have[k - 1][1] + c * (np.log(m) - np.log(have[k - 1][0])) + 0.01 * g
        have[k] = (m, g)
        lb.store(k, _t(m), _t(g))
    keep = min(ask, optimize.MAX_LBFGS_STORE)
    if any(k not in have for k in range(ask - keep, ask + 1)):
        with pytest.raises(Exception):
            lb.direction(ask)
        return
    d = lb.direction(ask).cpu().numpy()
    ref = orc.lbfgs_direction([have[k][0] for k in range(ask - keep, ask + 1)],
                              [have[k][1] for k in range(ask - keep, ask + 1)])
    assert np.abs(d - ref).max() <= 1e-11 * np.abs(ref).max()


def test_reductions_from_threads(gpu):
    """One context, many threads: each gets its own sums."""
    import threading
    import torch
    from surfattpp_b200 import optimize
    x = [torch.full((5000 + i,), float(i + 1), dtype=torch.float64, device="cuda:0")
         for i in range(6)]
    one = [torch.ones_like(v) for v in x]
    torch.cuda.synchronize()
    bad = []

    def run(i):
        for _ in range(50):
            if optimize.dot(x[i], one[i]) != (5000 + i) * (i + 1):
                bad.append(i)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("n", [1, 255, 257, GRID, GRID + 1])
def test_reductions(gpu, orc, n):
    from surfattpp_b200 import optimize
    rng = np.random.default_rng(n)
    x, y = rng.normal(size=n), rng.normal(size=n)
    assert abs(optimize.dot(_t(x), _t(y)) - float(np.dot(x, y))) <= 1e-13 * np.abs(x * y).sum()
    g = _t(x)
    m = optimize.grad_normalization(g)
    rg, rm = orc.grad_normalization(x)
    assert m == rm and np.array_equal(g.cpu().numpy(), rg)
