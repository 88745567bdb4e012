"""The encoder's kernels against the oracle, bit for bit, where they can go wrong: every
subspace width of the split kernels and the first one beyond, point counts around a block's
tile, equal codewords and values (the first wins), codewords a few roundings apart, and one-dimensional second quantizers whose
codewords repeat, lie far from the values, vanish, or are too large for the sorted search."""
import numpy as np
import pytest

import oracle
from puck_gb300 import native

pytestmark = pytest.mark.gpu


def _case(d, fnsq, pnsq, n, kind, seed=0):
    rng = np.random.default_rng(seed + d * 7 + fnsq + n)
    C, F = 5, 7
    if kind == "ties":  # small integers: equal distances everywhere
        draw = lambda *s: rng.integers(-2, 3, size=s).astype(np.float32)
    else:
        draw = lambda *s: rng.normal(size=s).astype(np.float32)
    a = dict(base=draw(n, d), coarse=draw(C, d), fine=draw(F, d),
             cell_assign=rng.integers(0, C * F, n).astype(np.uint32),
             filter_codebook=draw(fnsq, 256, d // fnsq),
             pq_codebook=draw(pnsq, 256, d // pnsq) if pnsq else None)
    if kind == "near":  # the order of two halves of a codebook is decided by the last bits
        for k in ("filter_codebook", "pq_codebook"):
            if a[k] is not None:
                a[k][:, 128:] = a[k][:, :128] * np.float32(1 + 2.0 ** -21)
    if kind == "far" and pnsq:
        a["pq_codebook"] += 50.0 * rng.normal(size=(pnsq, 1, 1)).astype(np.float32)
    if kind == "tiny":
        for k in ("base", "coarse", "fine", "filter_codebook", "pq_codebook"):
            if a[k] is not None:
                a[k] *= np.float32(1e-22)
    if kind == "huge" and pnsq:
        a["pq_codebook"][1, 17] = 3e18
        a["pq_codebook"][2, 5] = -2e19
        a["base"][0] = 1e19
    return a


@pytest.mark.parametrize("kind", ["normal", "ties", "near", "far", "tiny", "huge"])
@pytest.mark.parametrize("d,fnsq,pnsq", [(96, 24, 96), (30, 6, 30), (30, 5, 15), (16, 16, 4), (24, 12, 24),
                                         (21, 7, 3), (64, 8, 64), (18, 2, 18), (35, 5, 0), (40, 8, 40)])
def test_encode_shapes(d, fnsq, pnsq, kind):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    native.load(build_if_missing=True)
    for n in (1, 513, 1025):
        a = _case(d, fnsq, pnsq, n, kind)
        t = {k: None if v is None else torch.from_numpy(v.view(np.int32) if v.dtype == np.uint32 else v).cuda()
             for k, v in a.items()}
        got = native.puck_assign(t["base"], t["cell_assign"], t["coarse"], t["fine"],
                                 t["filter_codebook"], t["pq_codebook"])
        torch.cuda.synchronize()
        want = oracle.puck_assign(a["base"], a["cell_assign"], a["coarse"], a["fine"],
                                  a["filter_codebook"], a["pq_codebook"])
        for g, w in zip(got, want):
            if g is None:
                continue
            g = g.cpu().numpy()
            if g.dtype == np.float32:
                same = (g.view(np.uint32) == w.view(np.uint32)) | (np.isnan(g) & np.isnan(w))
                assert same.all()
            else:
                assert np.array_equal(g, w)
