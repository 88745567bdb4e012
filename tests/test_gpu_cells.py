"""The cell assignment's bounded search against the oracle, bit for bit, where it can go wrong:
fine counts around a group of 32, single clusters, points on a cell's centre (scores of 0 and
below, whose square root the walk's tests take), equal scores, fine centroids in no order of
norm, and a fine count whose group minima do not fit shared memory."""
import numpy as np
import pytest

import oracle
from puck_gb300 import native

pytestmark = pytest.mark.gpu


def _check(coarse, fine, x):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    native.load(build_if_missing=True)
    t = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda() for a in (coarse, fine, x)]
    cell = torch.empty(len(x), dtype=torch.int32, device="cuda")
    dist = torch.empty(len(x), dtype=torch.float32, device="cuda")
    native.nearest_cell_assign(*t, cell, dist)
    torch.cuda.synchronize()
    ocell, odist = oracle.nearest_cell_assign(coarse, fine, x)
    assert np.array_equal(cell.cpu().numpy().view(np.uint32), ocell)
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), odist.view(np.uint32))


@pytest.mark.parametrize("order", ["norm", "any"])
@pytest.mark.parametrize("kind", ["normal", "ints", "wide"])
@pytest.mark.parametrize("C,F", [(1, 1), (1, 33), (40, 31), (40, 32), (70, 65), (33, 1), (130, 200)])
def test_cells(C, F, kind, order):
    rng = np.random.default_rng(C * 1000 + F)
    d, n = 12, 700
    if kind == "ints":
        draw = lambda *s: rng.integers(-2, 3, size=s).astype(np.float32)
    else:
        draw = lambda *s: rng.normal(size=s).astype(np.float32)
    coarse, fine, x = draw(C, d), draw(F, d), draw(n, d)
    if kind == "wide":
        coarse, x = 100.0 * coarse, 100.0 * x
    x[:60] = coarse[rng.integers(0, C, 60)] + fine[rng.integers(0, F, 60)]
    if C > 2:
        coarse[2] = coarse[1]
    if order == "norm":
        fine = fine[np.argsort(-np.linalg.norm(fine, axis=1), kind="stable")]
    _check(coarse, np.ascontiguousarray(fine), x)


def test_cells_many_fine():
    rng = np.random.default_rng(0)
    fine = rng.normal(size=(210_000, 2)).astype(np.float32)
    fine = fine[np.argsort(-np.linalg.norm(fine, axis=1), kind="stable")]
    _check(rng.normal(size=(2, 2)).astype(np.float32), fine, rng.normal(size=(40, 2)).astype(np.float32))
