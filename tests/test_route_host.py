"""Host parts of the routing loop: the first-fit rounds against the definition
and the sparse copy of the usage array against the dense one."""
import numpy as np
import pytest
import torch

from orthoroute_b200.negotiate import _host_usage, disjoint_order


@pytest.mark.parametrize("n,span", [(1, 4), (2, 1), (70, 60), (300, 12)])
def test_first_fit_rounds(n, span):
    rng = np.random.default_rng(n)
    lo = rng.integers(0, 100, (n, 3))
    hi = lo + rng.integers(0, span, (n, 3))
    boxes = np.stack([lo[:, 0], hi[:, 0], lo[:, 1], hi[:, 1], lo[:, 2], hi[:, 2]], 1).astype(np.int32)
    idx = rng.permutation(n)
    rounds = []
    for i in idx:
        for r in rounds:
            if not any((lo[i] <= hi[k]).all() and (lo[k] <= hi[i]).all() for k in r):
                r.append(i)
                break
        else:
            rounds.append([i])
    assert disjoint_order(boxes, idx).tolist() == [i for r in rounds for i in r]


@pytest.mark.parametrize("n,used", [(1, 0), (64, 8), (64, 9), (5000, 40), (5000, 5000)])
def test_host_usage(n, used):
    u = torch.zeros(n, dtype=torch.int32)
    u[torch.randperm(n, generator=torch.Generator().manual_seed(n))[:used]] = torch.arange(1, used + 1, dtype=torch.int32)
    got = _host_usage(u)
    assert got.dtype == np.int32 and np.array_equal(got, u.numpy())
