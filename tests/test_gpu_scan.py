"""Scan mode's filter stage against the oracle's restatement, bit for bit, where its
paths change hands: every record kept or a sampled bound, buffers that overflow and
queries with more clusters than slots (both answered by the fused kernel), filter_topk
of 1, above the buffer of two blocks per SM, and above the records of the probed
clusters; rows of cell terms that are not whole float4s; groups of clusters. Then the rerank
of both modes: forms of the PQ table, and equal distances, whose order is the heap's.
"""
import os
import tempfile

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


def _index(tmp, n, d, C, F, nsq, seed, distinct, pq_nsq=0, equal=False, nq=70):
    import torch
    from puck_gb300 import builder
    base = builder.gmm(n, d, 64, "unit", seed)
    if distinct:
        base = base[torch.arange(n, device=base.device) % distinct].contiguous()
    a = builder.build_index(base, C, F, nsq, False, train_sample=min(n, 65536), iters=4,
                            pq_sample=min(n, 32768), seed=seed, whether_pq=pq_nsq > 0,
                            pq_nsq=pq_nsq or None)
    if equal:
        for c in (a["coarse"], a["fine"]):
            c[1::2] = c[0:len(c) - 1:2]
    index_io.write_index(tmp, base=a["base"], coarse=a["coarse"], fine=a["fine"],
                         cell_assign=a["cell_assign"], filter_codebook=a["filter_codebook"],
                         filter_offsets=a["filter_offsets"], filter_codes=a["filter_codes"],
                         whether_norm=False, pq_codebook=a.get("pq_codebook"),
                         pq_offsets=a.get("pq_offsets"), pq_codes=a.get("pq_codes"))
    return builder.gmm(nq, d, 64, "unit", seed, row_seed=seed + 7).cpu().numpy()


@pytest.mark.parametrize("n,d,C,F,nsq,P,T,distinct", [
    (30_000, 64, 12, 40, 16, 1, 100, 0),     # a few thousand records: all kept
    (60_000, 64, 12, 37, 16, 12, 1, 0),      # sampled, one candidate, odd rows
    (60_000, 64, 40, 33, 16, 40, 1500, 0),   # several groups of clusters
    (200_000, 32, 6, 50, 8, 6, 300, 0),      # several sampling passes
    (40_000, 64, 10, 4600, 16, 10, 2048, 0),  # one block per SM
    (9_000, 16, 5, 20, 4, 2, 2048, 0),       # close to all of the records, fewer for some
    (60_000, 32, 8, 16, 8, 8, 200, 150),     # 150 distinct vectors: ties fill the buffer
    (20_000, 32, 600, 10, 8, 600, 50, 0),    # more clusters than slots
    (40_000, 96, 16, 2000, 24, 16, 700, 0),  # two clusters to a group
])
def test_scan_matches_oracle(n, d, C, F, nsq, P, T, distinct):
    k = min(10, T)
    with tempfile.TemporaryDirectory() as tmp:
        q = _index(tmp, n, d, C, F, nsq, 5, distinct)
        ix = native.GpuIndex(tmp, search_coarse_count=P, filter_topk=T, topk=k, max_batch=64,
                             mode=native.PGPU_MODE_SCAN)
        dist, ids = ix.search(q, k)
        od, oi, st = oracle.OracleIndex(tmp).search_batch(q, k, P, T, topk_max=k,
                                                          nthreads=os.cpu_count(), scan=True)
        assert (st == 0).all()
        assert np.array_equal(dist.view(np.uint32), od.view(np.uint32))
        assert np.array_equal(ids, oi)


@pytest.mark.parametrize("n,C,P,distinct", [(60_000, 8, 8, 150), (9_000, 520, 520, 0)])
def test_fused_kernel_takes_several_queries_per_block(n, C, P, distinct):
    """Every query left to the fused kernel, and more of them than its blocks: by ties, by
    clusters (some of them empty)."""
    with tempfile.TemporaryDirectory() as tmp:
        q = _index(tmp, n, 32, C, 16, 8, 5, distinct, nq=1400)
        ix = native.GpuIndex(tmp, search_coarse_count=P, filter_topk=200, topk=10, max_batch=1400,
                             mode=native.PGPU_MODE_SCAN)
        dist, ids = ix.search(q, 10)
        od, oi, st = oracle.OracleIndex(tmp).search_batch(q, 10, P, 200, topk_max=10,
                                                          nthreads=os.cpu_count(), scan=True)
        assert (st == 0).all()
        assert np.array_equal(dist.view(np.uint32), od.view(np.uint32))
        assert np.array_equal(ids, oi)


@pytest.mark.parametrize("mode", [native.PGPU_MODE_EXACT, native.PGPU_MODE_SCAN])
@pytest.mark.parametrize("d,nsq,pq_nsq,T,k,distinct", [
    (64, 16, 64, 300, 10, 0),     # table of one-dimensional subspaces, whole 16-byte rows
    (36, 12, 36, 513, 100, 0),    # rows that are not
    (96, 24, 48, 200, 10, 0),     # subspaces of two dimensions
    (192, 24, 192, 3600, 10, 0),  # a table too large for shared memory (exact mode)
    (32, 8, 32, 1100, 100, 300),  # equal distances: the heap's own order, PQ
    (32, 8, 0, 700, 100, 200),    # and on the vectors
    (32, 8, 0, 65, 64, 40),       # a heap of as many as the candidates allow
    (30, 6, 0, 40, 1, 25),        # and of one
])
def test_rerank_matches_oracle(d, nsq, pq_nsq, T, k, distinct, mode):
    P = 6
    if mode == native.PGPU_MODE_SCAN:
        T = min(T, 2048)  # the scan's largest
    with tempfile.TemporaryDirectory() as tmp:
        q = _index(tmp, 20_000, d, 10, 24, nsq, 9, distinct, pq_nsq)
        ix = native.GpuIndex(tmp, search_coarse_count=P, filter_topk=T, topk=k, max_batch=64, mode=mode)
        dist, ids = ix.search(q, k)
        od, oi, st = oracle.OracleIndex(tmp).search_batch(q, k, P, T, topk_max=k,
                                                          nthreads=os.cpu_count(),
                                                          scan=mode == native.PGPU_MODE_SCAN)
        assert (st == 0).all()
        assert np.array_equal(dist.view(np.uint32), od.view(np.uint32))
        assert np.array_equal(ids, oi)


@pytest.mark.parametrize("C,F,P", [(40, 1, 40), (40, 2, 12), (130, 33, 100), (300, 300, 290)])
def test_equal_centroids_match_oracle(C, F, P):
    """Equal coarse and fine scores: the order of the clusters and cells is the heap's."""
    d, k = 32, 10
    with tempfile.TemporaryDirectory() as tmp:
        q = _index(tmp, 12_000, d, C, F, 8, 3, 0, equal=True)
        ix = native.GpuIndex(tmp, search_coarse_count=P, filter_topk=100, topk=k, max_batch=64,
                             mode=native.PGPU_MODE_EXACT)
        dist, ids = ix.search(q, k)
        assert ix.walk_counters()["coarse_window_fallbacks"] > 0
        od, oi, st = oracle.OracleIndex(tmp).search_batch(q, k, P, 100, topk_max=k,
                                                          nthreads=os.cpu_count())
        assert (st == 0).all()
        assert np.array_equal(dist.view(np.uint32), od.view(np.uint32))
        assert np.array_equal(ids, oi)
