"""The split scan's sampled bound against the oracle, bit for bit, where its buffers are tight:
fine clusters so many that the block of two per SM has no room for the sampled keys.
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


def _matches_oracle(tmp, ix, q, k, P, T):
    dist, ids = ix.search(q, k)
    od, oi, st = oracle.OracleIndex(tmp).search_batch(q, k, P, T, topk_max=k, nthreads=os.cpu_count(),
                                                      scan=True)
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
