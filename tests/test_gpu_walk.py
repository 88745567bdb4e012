"""The exact walk's warp replay against the oracle, where it can go wrong: heaps of every
shape around the five levels a round reads (one slot to several rounds), cells of more points
than the precomputed batch, probed clusters beyond one window, and equal distances.
"""
import os
import tempfile

import numpy as np
import pytest

import oracle
from puck_gb300 import builder, index_io, native

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.fixture(scope="module")
def indexes():
    """Index directories: many small cells; few cells of about 1250 points; many clusters."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    native.load(build_if_missing=True)
    with tempfile.TemporaryDirectory() as tmp:
        out = {}
        for name, n, C, F in (("small", 12000, 24, 40), ("big", 20000, 4, 4), ("wide", 12000, 300, 8)):
            base = builder.gmm(n, 16, 64, "int", 5)
            base[n // 2:n // 2 + 400] = base[:400]  # repeated rows: equal distances
            a = builder.build_index(base, C, F, 4, False, train_sample=n, iters=4, pq_sample=n, seed=5)
            index_io.write_index(os.path.join(tmp, name), whether_norm=False, **{
                k: a[k] for k in ("base", "coarse", "fine", "cell_assign", "filter_codebook",
                                  "filter_offsets", "filter_codes")})
            q = builder.gmm(96, 16, 64, "int", 5, row_seed=9).cpu().numpy()
            q[:32] = base[:32].cpu().numpy()
            out[name] = (os.path.join(tmp, name), q)
        yield out


@pytest.mark.parametrize("name", ["small", "big", "wide"])
@pytest.mark.parametrize("T", [1, 2, 3, 7, 31, 32, 62, 63, 64, 200, 1023, 1025, 2100, 4096])
def test_walk_heap_shapes(indexes, name, T):
    path, q = indexes[name]
    k = min(T, 20)
    P = 1000  # clamped to the index's clusters: every one is probed
    # the same queries as one pass of 192 blocks (more than SMs) and two of 96
    ix = native.GpuIndex(path, search_coarse_count=P, filter_topk=T, topk=k, max_batch=192)
    wide, wide_ids = ix.search(np.concatenate([q, q]), k)
    assert np.array_equal(_bits(wide[:96]), _bits(wide[96:])) and np.array_equal(wide_ids[:96], wide_ids[96:])
    dist, ids = ix.search(q, k)
    stats = ix.last_stats()
    assert np.array_equal(_bits(dist), _bits(wide[:96])) and np.array_equal(ids, wide_ids[:96])
    ix.close()
    orc = oracle.OracleIndex(path)
    od, oi, st = orc.search_batch(q, k, P, T, topk_max=k, nthreads=os.cpu_count())
    assert (st == 0).all()
    assert np.array_equal(_bits(dist), _bits(od))
    assert np.array_equal(ids, oi)
    traces = [orc.search_one(x, k, P, T, topk_max=k, trace=True)[4] for x in q]
    assert stats["cells_scanned"] == sum(t["scanned_cells"] for t in traces)
    assert stats["records_scanned"] == sum(t["scanned_points"] for t in traces)


@pytest.mark.parametrize("rate", [1.0, 1.3])
def test_walk_radius_rate(indexes, rate):
    path, q = indexes["small"]
    ix = native.GpuIndex(path, search_coarse_count=24, filter_topk=100, topk=10, radius_rate=rate,
                         max_batch=96)
    dist, ids = ix.search(q, 10)
    ix.close()
    od, oi, _ = oracle.OracleIndex(path).search_batch(q, 10, 24, 100, topk_max=10, radius_rate=rate,
                                                      nthreads=os.cpu_count())
    assert np.array_equal(_bits(dist), _bits(od)) and np.array_equal(ids, oi)
