"""The split scan's sampled bound against the oracle, bit for bit, where its buffers are tight:
fine clusters so many that the block of two per SM has no room for the sampled keys; records
inserted into a realtime index among the sampled ones; queries that it leaves to the fused
kernel (which alone counts the records it looked at, in the second counter).
"""
import os
import tempfile

import numpy as np
import pytest

import oracle
from puck_gb300 import native
from test_gpu_scan import _index

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    native.load(build_if_missing=True)


def _matches_oracle(tmp, ix, q, k, P, T, inserted=None):
    dist, ids = ix.search(q, k)
    orc = oracle.OracleIndex(tmp)
    if inserted is not None:
        orc.realtime_open()
        for x in inserted:
            orc.insert(x)
    od, oi, st = orc.search_batch(q, k, P, T, topk_max=k, nthreads=os.cpu_count(), scan=True)
    assert (st == 0).all()
    assert np.array_equal(dist.view(np.uint32), od.view(np.uint32))
    assert np.array_equal(ids, oi)


@pytest.mark.parametrize("d,F,C,P,T", [
    (16, 7400, 520, 512, 100),  # 768 keys in the block of two per SM
    (16, 6940, 520, 512, 1),    # 1004
    (4, 8192, 300, 300, 340),   # the largest
])
def test_many_fine_clusters_few_subspaces(d, F, C, P, T):
    with tempfile.TemporaryDirectory() as tmp:
        q = _index(tmp, 40_000, d, C, F, 4, 5, 0, nq=40)
        ix = native.GpuIndex(tmp, search_coarse_count=P, filter_topk=T, topk=min(10, T), max_batch=64,
                             mode=native.PGPU_MODE_SCAN)
        _matches_oracle(tmp, ix, q, min(10, T), P, T)


def _left(ix):
    """Records of all queries, and of those that the fused kernel answered."""
    c = ix.walk_counters()
    return c["records"], c["cells"]


@pytest.mark.parametrize("n,inserts,T", [(24_000, 9_000, 300), (3_000, 12_000, 40)])
def test_inserted_records_among_the_sampled(n, inserts, T):
    with tempfile.TemporaryDirectory() as tmp:
        q = _index(tmp, n, 32, 6, 16, 8, 5, 0)
        x = _index(tempfile.mkdtemp(dir=tmp), 2_000, 32, 4, 4, 8, 5, 0, nq=inserts)
        ix = native.GpuIndex(tmp, search_coarse_count=6, filter_topk=T, topk=10, max_batch=64,
                             mode=native.PGPU_MODE_SCAN)
        ix.realtime_open(inserts)
        ix.insert(x)
        _matches_oracle(tmp, ix, q, 10, 6, T, inserted=x)
        records, left = _left(ix)
        assert records >= 64 * (n + inserts) // 2 and left < records // 4


@pytest.mark.parametrize("distinct", [3, 5])
def test_equal_records_overflow_the_buffer(distinct):
    """More copies of each vector than the key buffer takes: every query is left."""
    with tempfile.TemporaryDirectory() as tmp:
        q = _index(tmp, 60_000, 32, 2, 4, 8, 5, distinct, nq=400)
        ix = native.GpuIndex(tmp, search_coarse_count=2, filter_topk=200, topk=10, max_batch=400,
                             mode=native.PGPU_MODE_SCAN)
        _matches_oracle(tmp, ix, q, 10, 2, 200)
        records, left = _left(ix)
        assert left == records == 400 * 60_000


def test_left_queries_with_many_rounds_per_cluster():
    """More clusters than slots and about 3800 records in each: every query is left, several
    per block, and each cluster takes more rounds of copies than the ring has stages."""
    with tempfile.TemporaryDirectory() as tmp:
        q = _index(tmp, 2_000_000, 32, 520, 8, 8, 5, 0, nq=330)
        ix = native.GpuIndex(tmp, search_coarse_count=520, filter_topk=200, topk=10, max_batch=330,
                             mode=native.PGPU_MODE_SCAN)
        _matches_oracle(tmp, ix, q, 10, 520, 200)
        records, left = _left(ix)
        assert left == records == 330 * 2_000_000
