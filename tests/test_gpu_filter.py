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
