"""Workloads that the library is timed on: searches through every mode and form, the serving
loop, the build's kernels and the learned probe's training.

A case is a dict of plain values; ``kind`` names the entry point it goes through:

  search   GpuIndex search: ``api`` one (search_one), host (search), device (search_device) or
           serve (one Server request); ``mode`` exact or scan; ``form`` fp32, bf16 or learned
           (probe + BF16); ``pq`` 1 for an index with the second-level PQ rerank
  assign   nearest_center, the assignment step of every k-means of a build
  cells    nearest_cell_assign, the build's exact cell assignment
  encode   puck_assign, the build's encoder
  train    Probe.train_step
  knn      knn, the labels of the probe's training set

Indexes are made here from seeded Gaussian mixtures (the families of the benchmark) with a few
Lloyd iterations in plain torch, so an index depends on its seed alone.
"""
import math

import numpy as np
import torch

from puck_gb300 import native

MIXTURE = {"unit": 0.3, "int": 12.0}  # per-dimension sigma of the two data families


def listed():
    return [
        # One caller asks for one query on an index opened with the defaults: exact mode,
        # search_coarse_count 200, filter_topk 1100, the second-level PQ rerank of the
        # reference's default index.
        dict(name="one_query", kind="search", api="one", mode="exact", form="fp32", pq=1, data="int",
             n=200_000, d=128, C=500, F=500, nsq=32, P=200, T=1100, k=10, nq=1),
        # The plain 1M x 128 integer configuration at its own settings, exact mode, host
        # buffers: an offline batch that has to return what the reference returns.
        dict(name="exact_batch", kind="search", api="host", mode="exact", form="fp32", pq=0,
             data="int", n=1_000_000, d=128, C=1000, F=1000, nsq=32, P=200, T=200, k=10, nq=10_000),
        # One request of uneven size through the serving loop (captured graphs, padded bucket).
        dict(name="served_request", kind="search", api="serve", mode="scan", form="fp32", pq=0,
             data="unit", n=1_000_000, d=96, C=500, F=500, nsq=24, P=2, T=500, k=100, nq=173),
        # The throughput path with the per-query work of the 100M configuration: 25k records
        # per coarse cluster, 4000 fine clusters, filter_topk 1100.
        dict(name="scan_batch", kind="search", api="device", mode="scan", form="fp32", pq=0,
             data="unit", n=5_000_000, d=96, C=200, F=4000, nsq=24, P=1, T=1100, k=10, nq=10_000),
        # The learned probe on the precision form, with the fixed count as its fallback.
        dict(name="learned_batch", kind="search", api="device", mode="scan", form="learned", pq=0,
             data="unit", n=5_000_000, d=96, C=1414, F=1414, nsq=24, P=200, T=500, k=10, nq=10_000),
        # Several clusters per query, an odd batch and long result lists on a PQ index.
        dict(name="pq_scan", kind="search", api="device", mode="scan", form="fp32", pq=1,
             data="unit", n=1_000_000, d=96, C=500, F=500, nsq=24, P=8, T=1100, k=100, nq=1537),
        # One assignment step of the coarse k-means on the builder's training sample.
        dict(name="kmeans_assign", kind="assign", data="unit", n=262_144, d=96, k=2000),
        # One assignment step of a filter-PQ codebook (256 codewords of a 4-dim subspace).
        dict(name="pq_kmeans", kind="assign", data="unit", n=131_072, d=4, k=256),
        # A build's exact cell assignment of a chunk of points.
        dict(name="cell_assign", kind="cells", data="unit", n=100_000, d=96, C=500, F=500),
        # The records of an index with both quantizers (filter PQ and one code per dimension).
        dict(name="encode", kind="encode", data="unit", n=500_000, d=96, C=1000, F=1000, nsq=24,
             pnsq=96),
        # Four optimizer steps of the probe network on batches of 2048, and its weights.
        dict(name="probe_train", kind="train", data="unit", d=96, h=512, C=4000, batch=2048, L=10,
             steps=4),
        # Labels of a batch of training queries: brute force over the indexed vectors.
        dict(name="knn_labels", kind="knn", data="unit", n=1_000_000, d=96, nq=2048, k=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform over the listed ranges, odd ones included."""
    kind = rng.choice(["search"] * 5 + ["assign"] * 2 + ["cells", "encode", "train", "knn"])
    data = rng.choice(["unit", "int"])
    if kind == "assign":
        if rng.random() < 0.4:
            return dict(kind=kind, data=data, n=_log_int(rng, 20_000, 131_072),
                        d=rng.choice([1, 2, 4, 5, 8]), k=256)
        return dict(kind=kind, data=data, n=_log_int(rng, 20_000, 262_144),
                    d=rng.choice([30, 64, 96, 100, 128]), k=_log_int(rng, 100, 2000))
    if kind == "cells":
        return dict(kind=kind, data=data, n=_log_int(rng, 10_000, 100_000),
                    d=rng.choice([30, 64, 96]), C=_log_int(rng, 100, 500), F=_log_int(rng, 100, 500))
    if kind == "encode":
        d, nsq = rng.choice([(96, 24), (128, 32), (64, 16), (30, 6), (96, 12)])
        return dict(kind=kind, data=data, n=_log_int(rng, 20_000, 300_000), d=d,
                    C=_log_int(rng, 100, 1000), F=_log_int(rng, 100, 1000), nsq=nsq,
                    pnsq=rng.choice([0, d, d // 2]))
    if kind == "train":
        return dict(kind=kind, data="unit", d=rng.choice([64, 96, 128]), h=rng.choice([256, 512]),
                    C=_log_int(rng, 200, 4000), batch=rng.choice([1000, 1024, 2048]),
                    L=rng.choice([1, 10]), steps=rng.choice([1, 2, 4]))
    if kind == "knn":
        return dict(kind=kind, data=data, n=_log_int(rng, 50_000, 1_000_000),
                    d=rng.choice([64, 96]), nq=_log_int(rng, 100, 2048), k=rng.choice([1, 10, 33, 64]))
    d, nsq = rng.choice([(96, 24), (128, 32), (64, 16), (96, 24), (48, 12), (30, 6)])
    mode = rng.choice(["exact", "scan", "scan", "scan"])
    api = rng.choice(["one", "host", "device", "device", "serve"])
    form = rng.choice(["fp32", "fp32", "bf16", "learned"]) if mode == "scan" else "fp32"
    data = "unit" if form == "learned" else data
    n = _log_int(rng, 100_000, 1_000_000)
    C, F = _log_int(rng, 100, 1000), _log_int(rng, 100, 1000)
    k = rng.choice([1, 10, 10, 100])
    P = min(C, 200 if mode == "exact" or form == "learned" else _log_int(rng, 1, 64))
    T = rng.choice([200, 500, 1100])
    nq = 1 if api == "one" else _log_int(rng, 1, 256) if api == "serve" else _log_int(rng, 16, 10_000)
    # no more records than the largest listed search scans
    per_query = max(1, n // C) * (2 if form == "learned" else P)
    if mode == "scan":
        nq = max(1, min(nq, 200_000_000 // per_query))
    elif nq > 2000:
        nq = 2000 + nq % 1000
    return dict(kind=kind, api=api, mode=mode, form=form, pq=int(form == "fp32" and rng.random() < 0.3),
                data=data, n=n, d=d, C=C, F=F, nsq=nsq, P=P, T=T, k=k, nq=nq)


# ------------------------------------------------------------------ data and indexes

def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(seed * 1009 + salt)


def _centers(case, g):
    m = 1024
    c = torch.rand(m, case["d"], generator=g, device="cuda") * 128 if case["data"] == "int" else \
        torch.randn(m, case["d"], generator=g, device="cuda")
    return c


def _rows(case, centers, n, g):
    """Rows of the mixture: integers in [0, 255], or unit vectors."""
    out = torch.empty(n, case["d"], device="cuda")
    for s in range(0, n, 1 << 20):
        m = min(1 << 20, n - s)
        pick = torch.randint(0, centers.shape[0], (m,), generator=g, device="cuda")
        x = centers[pick] + MIXTURE[case["data"]] * torch.randn(m, case["d"], generator=g, device="cuda")
        out[s:s + m] = x.clamp_(0, 255).round_() if case["data"] == "int" else \
            x / x.norm(dim=1, keepdim=True)
    return out


def _nearest(x, cents, chunk=1 << 18):
    half = 0.5 * (cents * cents).sum(1)
    out = torch.empty(x.shape[0], dtype=torch.int64, device=x.device)
    for s in range(0, x.shape[0], chunk):
        out[s:s + chunk] = torch.addmm(half, x[s:s + chunk], cents.T, alpha=-1.0).argmin(1)
    return out


def _lloyd(x, k, g, iters=4):
    cents = x[torch.randperm(x.shape[0], generator=g, device="cuda")[:k]].clone()
    for _ in range(iters):
        hot = torch.zeros(k, x.shape[0], device="cuda")
        hot[_nearest(x, cents), torch.arange(x.shape[0], device="cuda")] = 1.0
        cnt = hot.sum(1, keepdim=True)
        cents = torch.where(cnt > 0, hot @ x / cnt.clamp(min=1.0), cents)
    return cents


def _codebook(res, nsq, g):
    """[nsq, 256, lsq]: 256 codewords per subspace from a sample of residuals."""
    n, d = res.shape
    return torch.stack([_lloyd(res[:, m * (d // nsq):(m + 1) * (d // nsq)].contiguous(), 256, g, 3)
                        for m in range(nsq)])


def _encode(res, books):
    nsq, _, lsq = books.shape
    codes = torch.empty(res.shape[0], nsq, dtype=torch.uint8, device="cuda")
    for m in range(nsq):
        codes[:, m] = _nearest(res[:, m * lsq:(m + 1) * lsq].contiguous(), books[m], 1 << 20).to(torch.uint8)
    return codes


def _decode(codes, books):
    nsq, _, lsq = books.shape
    return torch.cat([books[m][codes[:, m].long()] for m in range(nsq)], 1)


def _index(case, seed):
    """The contents of an index's files (CUDA tensors, input order)."""
    g = _gen(seed, 1)
    centers = _centers(case, g)
    base = _rows(case, centers, case["n"], g)
    sample = base[torch.randperm(case["n"], generator=g, device="cuda")[:max(16384, 8 * case["C"])]]
    coarse = _lloyd(sample, case["C"], g)
    res = sample - coarse[_nearest(sample, coarse)]
    fine = _lloyd(res, case["F"], g)
    fine = fine[torch.argsort(-(fine * fine).sum(1), stable=True)].contiguous()
    res = (res - fine[_nearest(res, fine)])[:16384]
    books = _codebook(res, case["nsq"], g)
    cell = torch.empty(case["n"], dtype=torch.int64, device="cuda")
    codes = torch.empty(case["n"], case["nsq"], dtype=torch.uint8, device="cuda")
    offs = torch.empty(case["n"], device="cuda")
    ix = dict(base=base, coarse=coarse, fine=fine, filter_codebook=books, cell_assign=cell,
              filter_codes=codes, filter_offsets=offs, whether_norm=case["data"] == "unit",
              centers=centers)
    if case["pq"]:
        left = res - _decode(_encode(res, books), books)
        qs = (torch.arange(256, device="cuda") + 0.5) / 256
        levels = torch.quantile(left, qs, dim=0).T.contiguous()  # [d, 256] ascending
        ix.update(pq_codebook=levels[:, :, None].contiguous(),
                  pq_codes=torch.empty(case["n"], case["d"], dtype=torch.uint8, device="cuda"),
                  pq_offsets=torch.empty(case["n"], device="cuda"))
    for s in range(0, case["n"], 1 << 20):
        e = slice(s, min(s + (1 << 20), case["n"]))
        c = _nearest(base[e], coarse)
        r = base[e] - coarse[c]
        f = _nearest(r, fine)
        r = r - fine[f]
        cell[e] = c * case["F"] + f
        codes[e] = _encode(r, books)
        dec = _decode(codes[e], books)
        vocab = coarse[c] + fine[f]
        offs[e] = 2.0 * (dec * vocab).sum(1)
        if case["pq"]:
            mids = ((levels[:, 1:] + levels[:, :-1]) / 2).contiguous()
            pc = torch.searchsorted(mids, (r - dec).T.contiguous())  # [d, rows]
            ix["pq_codes"][e] = pc.T.to(torch.uint8)
            ix["pq_offsets"][e] = 2.0 * (torch.gather(levels, 1, pc).T * (vocab + dec)).sum(1)
    return ix


def _probe_weights(ix, case, h=512, beta=40.0):
    """W1, b1, W2, b2, W3, b3 of a network whose scores are beta (q.c - |c|^2 / 2), written
    with gelu(a) - gelu(-a) = a: what training on these mixtures converges to."""
    g = torch.Generator().manual_seed(case["d"] * 31 + h)
    s = 4.0 * torch.linalg.qr(torch.randn(h // 2, case["d"], generator=g))[0].cuda()
    proj = s @ s.T / 16.0
    w3 = beta * ix["coarse"] @ s.T / 16.0
    zero = torch.zeros(h, device="cuda")
    return (torch.cat([s, -s]), zero, torch.cat([torch.cat([proj, -proj], 1), torch.cat([-proj, proj], 1)]),
            zero, torch.cat([w3, -w3], 1), -beta * 0.5 * (ix["coarse"] * ix["coarse"]).sum(1))


def _queries(case, ix, seed):
    return _rows(case, ix["centers"], case["nq"], _gen(seed, 2))


def _max_probe(case):
    return min(8, case["C"])


# ------------------------------------------------------------------ prepare and run

def _prepare_search(case, seed):
    ix = _index(case, seed)
    q = _queries(case, ix, seed)
    arrays = {k: v.cpu().numpy() for k, v in ix.items() if torch.is_tensor(v) and k != "centers"}
    arrays["whether_norm"] = ix["whether_norm"]
    scan = case["mode"] == "scan"
    bf16 = case["form"] != "fp32"
    index = native.GpuIndex(
        arrays=arrays, search_coarse_count=case["P"], filter_topk=case["T"], topk=100,
        max_batch=max(case["nq"], 16), device=0,
        mode=native.PGPU_MODE_SCAN if scan else native.PGPU_MODE_EXACT,
        precision=native.PGPU_PRECISION_BF16 if bf16 else native.PGPU_PRECISION_FP32,
        filter_margin=case["T"] // 10 if bf16 else 0)
    st = dict(case=case, index=index)
    if case["form"] == "learned":
        st["probe"] = native.Probe(case["d"], 512, case["C"], seed=1)
        st["probe"].set_params(torch.cat([w.reshape(-1) for w in _probe_weights(ix, case)]).cpu().numpy())
        index.set_probe(st["probe"], mass=0.9, max_probe=_max_probe(case))
    if case["api"] == "device":
        st["q"] = q
        st["dist"] = torch.empty(case["nq"], case["k"], device="cuda")
        st["ids"] = torch.empty(case["nq"], case["k"], dtype=torch.int32, device="cuda")
    else:
        st["q"] = q.cpu().numpy()
    if case["api"] == "serve":
        st["server"] = native.Server(index, max_batch=256, scratch_budget_bytes=1 << 30, max_slots=2)
    return st


def _train_data(case, seed):
    """Training queries, the ids of the L nearest of C cluster centres each, initial weights."""
    g = _gen(seed, 3)
    centers = _centers(case, g)
    x = _rows(case, centers, case["batch"] * case["steps"], g)
    cents = _rows(case, centers, case["C"], g)
    labels = torch.topk(x @ cents.T, case["L"], dim=1).indices.to(torch.int32)
    d, h, C = case["d"], case["h"], case["C"]
    weights = torch.cat([w for rows, cols in ((h, d), (h, h), (C, h)) for w in (
        (2.0 * torch.rand(rows * cols, generator=g, device="cuda") - 1.0) * math.sqrt(3.0 / cols),
        torch.zeros(rows, device="cuda"))])
    return x, labels, weights


def _points(case, seed):
    g = _gen(seed, 3)
    centers = _centers(case, g)
    x = _rows(case, centers, case["n"], g)
    return x, centers, g


def _cells_data(case, seed):
    x, _, g = _points(case, seed)
    sample = x[:max(16384, 8 * case["C"])]
    coarse = _lloyd(sample, case["C"], g)
    fine = _lloyd(sample - coarse[_nearest(sample, coarse)], case["F"], g)
    return x, coarse, fine[torch.argsort(-(fine * fine).sum(1), stable=True)].contiguous()


def _encode_data(case, seed):
    x, coarse, fine = _cells_data(case, seed)
    c = _nearest(x, coarse)
    cell = torch.empty_like(c)
    for s in range(0, case["n"], 1 << 18):
        e = slice(s, s + (1 << 18))
        cell[e] = c[e] * case["F"] + _nearest(x[e] - coarse[c[e]], fine)
    g = _gen(seed, 5)
    res = (x - coarse[cell // case["F"]] - fine[cell % case["F"]])[:16384]
    books = _codebook(res, case["nsq"], g)
    pbooks = _codebook(res - _decode(_encode(res, books), books), case["pnsq"], g) if case["pnsq"] else None
    return x, cell.to(torch.int32), coarse, fine, books, pbooks


def _assign_data(case, seed):
    x, _, g = _points(case, seed)
    return x, _lloyd(x[:max(16384, 8 * case["k"])], case["k"], g, 2)


def _knn_data(case, seed):
    x, centers, g = _points(case, seed)
    return x, _rows(case, centers, case["nq"], g)


def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "search":
        return _prepare_search(case, seed)
    st = dict(case=case)
    if kind == "assign":
        st["x"], st["cents"] = _assign_data(case, seed)
        st["assign"] = torch.empty(n, dtype=torch.int32, device="cuda")
        st["dist"] = torch.empty(n, device="cuda")
    elif kind == "cells":
        st["x"], st["coarse"], st["fine"] = _cells_data(case, seed)
        st["cell"] = torch.empty(n, dtype=torch.int32, device="cuda")
        st["dist"] = torch.empty(n, device="cuda")
    elif kind == "encode":
        st["args"] = _encode_data(case, seed)
    elif kind == "train":
        x, lab, weights = _train_data(case, seed)
        b = case["batch"]
        st["batches"] = [(x[i * b:(i + 1) * b].contiguous(), lab[i * b:(i + 1) * b].contiguous())
                         for i in range(case["steps"])]
        st["probe"] = native.Probe(case["d"], case["h"], case["C"], seed=1)
        st["probe"].set_params(weights.cpu().numpy())
        torch.cuda.synchronize()
    else:
        st["x"], st["q"] = _knn_data(case, seed)
        st["ids"] = torch.empty(case["nq"], case["k"], dtype=torch.int32, device="cuda")
        st["dist"] = torch.empty(case["nq"], case["k"], device="cuda")
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "search":
        k, api = case["k"], case["api"]
        if api == "device":
            st["index"].search_device(case["nq"], st["q"], k, st["dist"], st["ids"],
                                      stream=torch.cuda.current_stream())
            return dict(dist=st["dist"], ids=st["ids"])
        if api == "one":
            dist, ids, num = st["index"].search_one(st["q"][0], k)
            return dict(dist=dist, ids=ids.view(np.int32), num=num)
        if api == "serve":
            dist, ids, status, _ = st["server"].wait(st["server"].submit(st["q"], k))
            return dict(dist=dist, ids=ids.view(np.int32), status=status)
        dist, ids = st["index"].search(st["q"], k)
        return dict(dist=dist, ids=ids.view(np.int32))
    stream = torch.cuda.current_stream()
    if kind == "assign":
        native.nearest_center(st["cents"], st["x"], st["assign"], st["dist"], stream=stream)
        return dict(assign=st["assign"], dist=st["dist"])
    if kind == "cells":
        native.nearest_cell_assign(st["coarse"], st["fine"], st["x"], st["cell"], st["dist"], stream=stream)
        return dict(cell=st["cell"], dist=st["dist"])
    if kind == "encode":
        offs, codes, poffs, pcodes = native.puck_assign(*st["args"], stream=stream)
        out = dict(offsets=offs, codes=codes)
        return dict(out, pq_offsets=poffs, pq_codes=pcodes) if case["pnsq"] else out
    if kind == "train":
        losses = [st["probe"].train_step(x, lab, 1e-3) for x, lab in st["batches"]]
        return dict(loss=np.array(losses, np.float32), params=st["probe"].get_params())
    native.knn(st["x"], st["q"], case["k"], st["ids"], st["dist"], stream=stream)
    return dict(ids=st["ids"], dist=st["dist"])


# ------------------------------------------------------------------ least work

def work(case):
    """Bytes and operations of one pass: each input read once, each output written once; the
    distances the method has to form (a multiply and an add per dimension)."""
    kind, d = case["kind"], case["d"]
    if kind == "assign":
        n, k = case["n"], case["k"]
        return dict(bytes=4 * d * (n + k) + 8 * n, flops=2 * n * k * d)
    if kind == "cells":
        n, m = case["n"], case["C"] + case["F"]
        return dict(bytes=4 * d * (n + m) + 8 * n, flops=2 * n * m * d)
    if kind == "encode":
        n, codes = case["n"], case["nsq"] + case["pnsq"]
        quant = 2 if case["pnsq"] else 1
        return dict(bytes=n * (4 * d + 4 + codes + 4 * quant) + 4 * d * (case["C"] + case["F"] + 256 * quant),
                    flops=2 * n * 256 * d * quant)
    if kind == "train":
        h, C, steps = case["h"], case["C"], case["steps"]
        weights = h * d + h * h + C * h + 2 * h + C
        return dict(bytes=steps * (case["batch"] * 4 * (d + case["L"]) + 24 * weights) + 4 * weights,
                    flops=steps * 6 * case["batch"] * (h * d + h * h + C * h))
    if kind == "knn":
        n, nq = case["n"], case["nq"]
        return dict(bytes=4 * d * (n + nq) + 8 * nq * case["k"], flops=2 * n * nq * d)
    nq, P = case["nq"], case["P"] if case["form"] != "learned" else 1
    per = P * case["n"] // case["C"]  # records of a query's clusters
    rec = case["nsq"] + 6
    if case["mode"] == "exact":
        per = min(per, 4 * case["T"])  # the pivot ends most cells early
    rows = min(nq * case["T"], case["n"])
    row = (d + 4) if case["pq"] else 4 * d
    touched = min(nq * per, case["n"])
    return dict(bytes=4 * nq * d + touched * rec + rows * row + 8 * nq * case["k"] +
                4 * d * (case["C"] + case["F"]),
                flops=nq * (2 * d * (case["C"] + case["F"]) + per * case["nsq"] + 3 * case["T"] * d +
                            2 * 256 * d))


# ------------------------------------------------------------------ values in 64 bits

def _clusters64(case, ix, q, coarse):
    """Per query the probed clusters of a scan-mode search (list of id tensors)."""
    score = 0.5 * (coarse * coarse).sum(1)[None, :] - q @ coarse.T
    fixed = torch.topk(score, min(case["P"], case["C"]), dim=1, largest=False).indices
    if case["form"] != "learned":
        return list(fixed)
    w1, b1, w2, b2, w3, b3 = (w.double() for w in _probe_weights(ix, case))
    gelu = torch.nn.functional.gelu
    prob = torch.softmax(gelu(gelu(q @ w1.T + b1) @ w2.T + b2) @ w3.T + b3, 1)
    top = torch.topk(prob, _max_probe(case), dim=1)
    count = (torch.cumsum(top.values, 1) < 0.9).sum(1).tolist()
    return [top.indices[i, :c + 1] if c < _max_probe(case) else fixed[i] for i, c in enumerate(count)]


def _scan64(case, seed):
    """Distances of a scan-mode search: every record of the probed clusters, the filter_topk
    smallest filter distances, their exact (or second-level PQ) distances, the k smallest."""
    ix = _index(case, seed)
    q = _queries(case, ix, seed).double()
    if ix["whether_norm"]:
        q = q / q.norm(dim=1, keepdim=True)
    coarse, fine, base = ix["coarse"].double(), ix["fine"].double(), ix["base"]
    order = torch.argsort(ix["cell_assign"], stable=True)
    cell = ix["cell_assign"][order]
    bound = torch.searchsorted(cell // case["F"], torch.arange(case["C"] + 1, device="cuda")).tolist()
    fid = cell % case["F"]
    nsq = case["nsq"]
    slot = ix["filter_codes"][order].long() + 256 * torch.arange(nsq, device="cuda")
    offs = ix["filter_offsets"][order].double()
    books = ix["filter_codebook"].double()
    stat = 0.5 * (fine * fine).sum(1)[None, :] + coarse @ fine.T
    keep = case["T"] + (case["T"] // 10 if case["form"] != "fp32" else 0)
    out = torch.empty(case["nq"], case["k"], dtype=torch.float64, device="cuda")
    for i, clusters in enumerate(_clusters64(case, ix, q, coarse)):
        qi = q[i]
        table = ((qi.view(nsq, 1, -1) - books) ** 2).sum(2).reshape(-1)
        qf = fine @ qi
        rec, ts = [], []
        for c in clusters.tolist():
            a, b = bound[c], bound[c + 1]
            if a == b:
                continue
            term = 0.5 * (coarse[c] @ coarse[c]) - qi @ coarse[c] + stat[c] - qf
            ts.append(2.0 * term[fid[a:b]] + offs[a:b] + table[slot[a:b]].sum(1))
            rec.append(order[a:b])
        t, rec = torch.cat(ts), torch.cat(rec)
        t, at = torch.topk(t, min(keep, t.shape[0]), largest=False)
        rec = rec[at]
        if case["pq"]:
            levels = ix["pq_codebook"].double()[:, :, 0]
            dec = torch.gather(levels, 1, ix["pq_codes"][rec].long().T).T
            dist = t - qi @ qi + ix["pq_offsets"][rec].double() + ((qi - dec) ** 2).sum(1)
        else:
            dist = ((base[rec].double() - qi) ** 2).sum(1)
        got = torch.sort(dist).values[:case["k"]]
        out[i, :got.shape[0]] = got
        out[i, got.shape[0]:] = 3.3961514e38
    return out


def _assign64(x, cents, chunk=8192):
    c = cents.double()
    half = 0.5 * (c * c).sum(1)
    return torch.cat([((p := x[s:s + chunk].double()) * p).sum(1) + 2.0 * (half - p @ c.T).min(1).values
                      for s in range(0, x.shape[0], chunk)])


def _cells64(x, coarse, fine, chunk=256):
    c, f = coarse.double(), fine.double()
    stat = (0.5 * (f * f).sum(1)[None, :] + c @ f.T)
    half = 0.5 * (c * c).sum(1)
    out = []
    for s in range(0, x.shape[0], chunk):
        p = x[s:s + chunk].double()
        term = half - p @ c.T + 0.5 * (p * p).sum(1, keepdim=True)
        out.append((stat[None] - (p @ f.T)[:, None, :]).min(2).values.add_(term).min(1).values)
    return torch.cat(out)


def _encode64(case, seed):
    x, cell, coarse, fine, books, pbooks = _encode_data(case, seed)
    offs, poffs = [], []
    for s in range(0, case["n"], 1 << 16):
        ce = cell[s:s + (1 << 16)].long()
        c, f = coarse[ce // case["F"]].double(), fine[ce % case["F"]].double()
        r, v = x[s:s + (1 << 16)].double() - c - f, c + f
        for bk, to in ((books, offs), (pbooks, poffs)):
            if bk is None:
                continue
            bd, lsq = bk.double(), bk.shape[2]
            dec = torch.cat([bd[m][(0.5 * (bd[m] * bd[m]).sum(1) - r[:, m * lsq:(m + 1) * lsq] @ bd[m].T)
                                   .argmin(1)] for m in range(bk.shape[0])], 1)
            to.append(2.0 * (dec * v).sum(1))
            r, v = r - dec, v + dec
    out = dict(offsets=torch.cat(offs), codes=None)
    return dict(out, pq_offsets=torch.cat(poffs), pq_codes=None) if case["pnsq"] else out


def _train64(case, seed):
    x, lab, weights = _train_data(case, seed)
    flat = weights.double()
    d, h, C, b = case["d"], case["h"], case["C"], case["batch"]
    gelu = torch.nn.functional.gelu
    m, v, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
    for i in range(case["steps"]):
        p = flat.clone().requires_grad_(True)
        w1, b1, w2, b2, w3, b3 = torch.split(p, [h * d, h, h * h, h, C * h, C])
        y = gelu(x[i * b:(i + 1) * b].double() @ w1.view(h, d).T + b1)
        z = gelu(y @ w2.view(h, h).T + b2) @ w3.view(C, h).T + b3
        loss = -torch.log_softmax(z, 1).gather(1, lab[i * b:(i + 1) * b].long()).mean()
        grad, = torch.autograd.grad(loss, p)
        m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
        flat = flat - 1e-3 * (m / (1 - 0.9 ** (i + 1))) / ((v / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
        losses.append(float(loss))
    return dict(loss=np.array(losses), params=flat)


def _knn64(case, seed):
    x, q = _knn_data(case, seed)
    qd = q.double()
    best = torch.full((case["nq"], case["k"]), float("inf"), dtype=torch.float64, device="cuda")
    for s in range(0, case["n"], 1 << 16):
        p = x[s:s + (1 << 16)].double()
        dist = (qd * qd).sum(1, keepdim=True) + (p * p).sum(1) - 2.0 * qd @ p.T
        both = torch.cat([best, torch.topk(dist, min(case["k"], dist.shape[1]), 1, largest=False).values], 1)
        best = torch.topk(both, case["k"], 1, largest=False).values
    return dict(ids=None, dist=best)


def exact(case, seed):
    kind = case["kind"]
    if kind == "search":
        if case["mode"] == "exact":
            return None  # a walk whose result depends on its order, record by record
        out = dict(dist=_scan64(case, seed).cpu().numpy(), ids=None)
        if case["api"] == "one":
            out["num"] = None
        if case["api"] == "serve":
            out["status"] = None
        return out
    if kind == "assign":
        return dict(assign=None, dist=_assign64(*_assign_data(case, seed)))
    if kind == "cells":
        return dict(cell=None, dist=_cells64(*_cells_data(case, seed)))
    if kind == "encode":
        return _encode64(case, seed)
    return _train64(case, seed) if kind == "train" else _knn64(case, seed)
