"""The selecting contraction (tc_filter.cu) behind nearest_center and knn, where it can go wrong:
row, column and dimension counts around its tiles (128, 256, 64), equal scores, and rows or
centroids too large for the screen's bound."""
import numpy as np
import pytest

import oracle
from puck_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    native.load(build_if_missing=True)


def _nearest(cents, x):
    import torch
    a = torch.empty(len(x), dtype=torch.int32, device="cuda")
    d = torch.empty(len(x), dtype=torch.float32, device="cuda")
    native.nearest_center(torch.from_numpy(cents).cuda(), torch.from_numpy(x).cuda(), a, d,
                          stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    return a.cpu().numpy(), d.cpu().numpy()


@pytest.mark.parametrize("kind", ["normal", "ints", "offset"])
@pytest.mark.parametrize("n,k,d", [(1, 1, 1), (127, 31, 2), (129, 33, 4), (128, 256, 8), (300, 257, 63),
                                   (257, 255, 65), (500, 700, 96), (130, 513, 128), (200, 300, 250),
                                   (64, 40, 256), (64, 40, 257), (20000, 300, 30)])
def test_nearest_center_tiles(n, k, d, kind):
    rng = np.random.default_rng(n * 7 + k * 3 + d)
    if kind == "ints":
        draw = lambda *s: rng.integers(0, 4, size=s).astype(np.float32)
    else:
        draw = lambda *s: rng.normal(size=s).astype(np.float32) + np.float32(200 if kind == "offset" else 0)
    cents, x = draw(k, d), draw(n, d)
    if k > 3:
        cents[3] = cents[1]
    x[: n // 4] = cents[rng.integers(0, k, n // 4)]
    a, dd = _nearest(cents, x)
    oa, od = oracle.nearest_center(cents, x)
    assert np.array_equal(a, oa)
    assert np.array_equal(dd.view(np.uint32), od.view(np.uint32))


def test_nearest_center_beyond_the_bound():
    rng = np.random.default_rng(3)
    cents, x = rng.normal(size=(300, 24)).astype(np.float32), rng.normal(size=(200, 24)).astype(np.float32)
    x[5] *= np.float32(1e18)
    x[6] = np.float32(2e19)
    big = cents.copy()
    big[7] *= np.float32(1e19)
    for c in (cents, big):
        a, dd = _nearest(c, x)
        oa, od = oracle.nearest_center(c, x)
        assert np.array_equal(a, oa)
        assert np.array_equal(dd.view(np.uint32), od.view(np.uint32))


def _knn(base, q, k):
    import torch
    ids = torch.empty((len(q), k), dtype=torch.int32, device="cuda")
    dist = torch.empty((len(q), k), dtype=torch.float32, device="cuda")
    native.knn(torch.from_numpy(base).cuda(), torch.from_numpy(q).cuda(), k, ids, dist)
    torch.cuda.synchronize()
    return ids.cpu().numpy().view(np.uint32), dist.cpu().numpy()


def _knn_want(base, q, k):
    """Small integers: screened scores and distances are exact, so the result is the k
    smallest (distance, id)."""
    d2 = ((q * q).sum(1)[:, None] + (base * base).sum(1)[None] - 2.0 * q @ base.T).astype(np.float64)
    order = np.argsort(d2, axis=1, kind="stable")[:, :k]
    return order, np.take_along_axis(d2, order, 1)


@pytest.mark.parametrize("n,nq,d,k", [(1, 1, 1, 1), (63, 5, 8, 10), (255, 127, 3, 64), (257, 129, 30, 33),
                                      (2048, 300, 96, 10), (2049, 20, 16, 64), (30000, 260, 20, 64),
                                      (70001, 40, 96, 10), (3000, 33, 256, 10), (3000, 33, 257, 10)])
def test_knn_tiles(n, nq, d, k):
    rng = np.random.default_rng(n + nq)
    base = rng.integers(0, 4, size=(n, d)).astype(np.float32)
    q = rng.integers(0, 4, size=(nq, d)).astype(np.float32)
    ids, dist = _knn(base, q, min(k, n))
    want, wd = _knn_want(base, q, min(k, n))
    assert np.array_equal(ids, want)
    assert np.array_equal(dist, wd)


@pytest.mark.parametrize("order", ["sorted", "equal"])
def test_knn_crowded_lists(order):
    """Rows in runs of near copies, and all rows equal: more rows below a threshold than a list
    holds."""
    rng = np.random.default_rng(1)
    if order == "equal":
        base = np.ones((20000, 16), np.float32)
    else:
        base = np.repeat(rng.integers(0, 4, size=(6, 16)), 5000, axis=0).astype(np.float32)
        base[:, 0] += np.arange(30000) % 3
    q = rng.integers(0, 4, size=(50, 16)).astype(np.float32)
    ids, dist = _knn(base, q, 64)
    want, wd = _knn_want(base, q, 64)
    assert np.array_equal(ids, want)
    assert np.array_equal(dist, wd)
