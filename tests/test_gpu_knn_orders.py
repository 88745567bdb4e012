"""Brute-force neighbours over a base in any order: the same rows, whatever tiles of the base
lie near a query, and no order that costs a second pass.
"""
import time

import numpy as np
import pytest

from puck_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    native.load(build_if_missing=True)


def _mixture(n, d, nq, run, seed):
    """Base rows in the order of their clusters, `run` rows each, and queries near them."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    m = (n + run - 1) // run
    c = torch.randn(m, d, generator=g, device="cuda")
    base = c[torch.arange(n, device="cuda") // run] + 0.3 * torch.randn(n, d, generator=g, device="cuda")
    q = c[torch.randint(0, m, (nq,), generator=g, device="cuda")] + \
        0.3 * torch.randn(nq, d, generator=g, device="cuda")
    return base, q, torch.randperm(n, generator=g, device="cuda")


def _knn(base, q, k):
    import torch
    ids = torch.empty(q.shape[0], k, dtype=torch.int32, device="cuda")
    dist = torch.empty(q.shape[0], k, device="cuda")
    native.knn(base, q, k, ids, dist)
    return ids.cpu().numpy(), dist.cpu().numpy()


@pytest.mark.parametrize("n,d,nq,run,k", [
    (300_000, 96, 700, 1000, 10),   # a few tiles per cluster
    (300_000, 96, 1, 40_000, 10),   # clusters of more rows than the first columns
    (200_000, 30, 129, 128, 5),     # one half tile each
    (150_000, 256, 2500, 5000, 3),
    (100_003, 8, 40, 50_000, 1),    # nearly every row of a tile below the threshold
    (30_000, 16, 20_000, 10_000, 10),
])
def test_order_of_the_base(n, d, nq, run, k):
    base, q, perm = _mixture(n, d, nq, run, n + d)
    ids, dist = _knn(base, q, k)
    shuffled, dist2 = _knn(base[perm].contiguous(), q, k)
    assert np.array_equal(dist.view(np.uint32), dist2.view(np.uint32))
    assert (ids == perm.cpu().numpy()[shuffled]).all()


def test_runs_of_equal_rows():
    """The lowest ids of many equal rows."""
    import torch
    rows, q, _ = _mixture(40, 64, 40, 1, 7)
    base = rows.repeat_interleave(3000, dim=0).contiguous()
    near = torch.cdist(q.double(), rows.double()).argmin(1).cpu().numpy()
    ids, _ = _knn(base, q, 10)
    assert np.array_equal(ids, near[:, None] * 3000 + np.arange(10))


def test_no_order_costs_a_second_pass():
    """Sorted by cluster against shuffled: the selecting passes are a tenth of a pass with the
    screen in memory, so a repeated call shows as ten times the time."""
    import torch
    base, q, perm = _mixture(500_000, 96, 512, 1000, 3)
    took = []
    for b in (base[perm].contiguous(), base):
        best = float("inf")
        for _ in range(5):
            torch.cuda.synchronize()
            t = time.perf_counter()
            _knn(b, q, 10)
            best = min(best, time.perf_counter() - t)
        took.append(best)
    assert took[1] < 4 * took[0], took
