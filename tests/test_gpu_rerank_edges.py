"""The precision form's rerank at the smallest heap: one dimension and as few candidates as
results, where the heap's entries outnumber the slots of the sort keys.
"""
import numpy as np
import pytest

import oracle
from puck_gb300 import index_io, native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    native.load(build_if_missing=True)


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("T,k", [(1, 1), (2, 1), (2, 2), (3, 2), (4, 4)])
def test_few_candidates_few_dimensions(tmp_path, d, T, k):
    """Clusters of T points each, so that every record of the probed cluster is a candidate
    and the result does not depend on the filter's precision."""
    rng = np.random.default_rng(d * 10 + T)
    C = 6
    coarse = (20.0 * np.arange(C)[:, None] * np.ones((1, d))).astype(np.float32)
    fine = np.zeros((1, d), np.float32)
    cell = np.repeat(np.arange(C, dtype=np.uint32), T)
    res = rng.uniform(-1, 1, (C * T, d)).astype(np.float32)
    base = coarse[cell] + res
    books = rng.uniform(-1, 1, (d, 256, 1)).astype(np.float32)
    codes = np.stack([np.abs(res[:, m:m + 1] - books[m].T).argmin(1) for m in range(d)], 1).astype(np.uint8)
    dec = np.stack([books[m, codes[:, m], 0] for m in range(d)], 1)
    offs = (2.0 * (dec * coarse[cell]).sum(1)).astype(np.float32)
    index_io.write_index(str(tmp_path), base=base, coarse=coarse, fine=fine, cell_assign=cell,
                         filter_codebook=books, filter_offsets=offs, filter_codes=codes,
                         whether_norm=False)
    q = (coarse[rng.integers(0, C, 40)] + rng.uniform(-1, 1, (40, d))).astype(np.float32)
    ix = native.GpuIndex(str(tmp_path), search_coarse_count=1, filter_topk=T, topk=k, max_batch=64,
                         mode=native.PGPU_MODE_SCAN, precision=native.PGPU_PRECISION_BF16)
    dist, ids = ix.search(q, k)
    od, oi, st = oracle.OracleIndex(str(tmp_path)).search_batch(q, k, 1, T, topk_max=k, scan=True)
    assert (st == 0).all()
    assert np.array_equal(ids, oi)
    assert np.array_equal(dist.view(np.uint32), od.view(np.uint32))
