"""L-BFGS iterates numbered up to the largest int: the same direction, bit for
bit, as for small numbers, although the iterate after the last has none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_largest_iterates(gpu):
    import torch
    from surfattpp_b200 import optimize
    n, last = 1000, 2**31 - 1
    rng = np.random.default_rng(3)
    t = lambda a: torch.as_tensor(a, device="cuda:0")
    its = [(t(np.exp(rng.normal(1.2, 0.05, n))), t(rng.normal(size=n))) for _ in range(6)]
    out = []
    for top in (17, last):
        lb = optimize.LBFGS(n)
        for k, (m, g) in enumerate(its):
            lb.store(top - 5 + k, m, g)
        lb.store(top, *its[5])
        out.append(lb.direction(top))
    assert torch.equal(out[0], out[1])
