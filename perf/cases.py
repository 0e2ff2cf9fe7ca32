"""Timed search cases over indexes of several sizes, through the library's public entry points.

Every case opens an NGT index (built here on the GPU from fixed seeds and kept in the
temporary directory between processes) and searches it with queries made from the
case's seed: single queries and batches, host and device buffers, the exact-order and
the batched graph kernels, the plain and the tensor-core exhaustive searches, the
quantized graph and the quantized blob graph.

The indexes hold the data of the benchmark (coordinates min(255, rint(Exponential(25)))),
points of low intrinsic dimension in bytes (as image descriptors are), unit vectors of
low intrinsic dimension (as word embeddings are) and Gaussian clusters.
"""
from __future__ import annotations

import ctypes
import math
import os
import shutil
import struct
import tempfile

import numpy as np
import torch

from ngt_gb300 import qg_build
from ngt_gb300.base import (KERNEL_EXACT, KERNEL_WIDE, QBG_REFINE, QBG_TWO_STEP, Index, QBGIndex, QGQueryParameters,
                            QuantizedIndex)

# Batched-kernel settings: "throughput" is what the library's autotuner picks on the
# 1M x 128 benchmark index, "latency" what the serving loop uses, "default" untouched.
TUNINGS = {
    "throughput": dict(list_capacity=256, parents=10, cta_threads=128, stage_kilobytes=16),
    "latency": dict(parents=32),
    "default": {},
}


def listed():
    return [
        # one interactive query through the reference's C API on the benchmark index
        {"name": "graph one query 1M", "op": "graph_one", "data": "exponential", "rows": 1_000_000, "dim": 128,
         "queries": 1, "k": 20, "epsilon": 0.1},
        # a batch job that needs the reference's own results (exact order)
        {"name": "graph exact 1M", "op": "graph_exact", "data": "exponential", "rows": 1_000_000, "dim": 128,
         "queries": 2000, "k": 10, "epsilon": 0.08},
        # the benchmark's headline: 10,000 queries resident on the GPU, batched kernel
        {"name": "graph batched 1M", "op": "graph_wide", "data": "exponential", "rows": 1_000_000, "dim": 128,
         "queries": 10_000, "k": 10, "epsilon": 0.08, "tuning": "throughput", "host": False},
        # a small request as a server sees it: host buffers, latency settings, k = 100
        {"name": "graph request 1M", "op": "graph_wide", "data": "exponential", "rows": 1_000_000, "dim": 128,
         "queries": 17, "k": 100, "epsilon": 0.06, "tuning": "latency", "host": True},
        # embeddings under the cosine distance, a dimension that is no multiple of 16
        {"name": "graph cosine 200k", "op": "graph_wide", "data": "unit", "rows": 200_000, "dim": 100,
         "queries": 1500, "k": 20, "epsilon": 0.1, "tuning": "default", "host": True},
        # exhaustive search of one query through the reference's C API (ground truth, filters)
        {"name": "linear one query 1M", "op": "linear_one", "data": "clusters", "rows": 1_000_000, "dim": 768,
         "queries": 1, "k": 100},
        # the benchmark's exhaustive search: 10,000 queries resident on the GPU
        {"name": "linear tensor 1M", "op": "linear_tc", "data": "clusters", "rows": 1_000_000, "dim": 768,
         "queries": 10_000, "k": 100, "candidates": 400, "ties": True, "host": False},
        # exhaustive search of a request's queries from host buffers
        {"name": "linear tensor request", "op": "linear_tc", "data": "clusters", "rows": 1_000_000, "dim": 768,
         "queries": 33, "k": 10, "candidates": 0, "ties": False, "host": True},
        # exhaustive search with ragged sizes: L2 over descriptors, odd counts throughout
        {"name": "linear tensor ragged", "op": "linear_tc", "data": "bytes", "rows": 151_003, "dim": 100,
         "queries": 1501, "k": 20, "candidates": 0, "ties": False, "host": False},
        # quantized graph in the reference's order, as ngtpy's QuantizedIndex is used
        {"name": "quantized graph exact", "op": "qg_exact", "data": "bytes", "rows": 200_000, "dim": 128,
         "queries": 2000, "k": 20, "epsilon": 0.03, "expansion": 3.0},
        # quantized graph, relaxed order: a large batch resident on the GPU
        {"name": "quantized graph batched", "op": "qg_relaxed", "data": "bytes", "rows": 200_000, "dim": 128,
         "queries": 10_000, "k": 10, "epsilon": 0.02, "expansion": 10.0},
        # quantized blob graph: two-step search with exact refinement, as the CLI searches
        {"name": "blob graph two-step", "op": "qbg", "data": "bytes", "rows": 1_000_000, "dim": 128,
         "queries": 3000, "k": 10, "probes": 64, "expansion": 10.0, "two_step": True},
    ]


def _between(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["graph_one", "graph_exact", "graph_wide", "graph_wide", "linear_one", "linear_tc", "linear_tc",
                     "qg_exact", "qg_relaxed", "qbg"])
    if op in ("graph_one", "graph_exact", "graph_wide"):
        c = {"op": op, "data": rng.choice(["exponential", "bytes", "unit"]), "rows": _between(rng, 20_000, 400_000),
             "dim": _between(rng, 24, 200), "queries": 1, "k": _between(rng, 1, 100),
             "epsilon": round(rng.uniform(0.0, 0.12), 3)}
        if op == "graph_exact":
            c["queries"] = _between(rng, 2, 2500)
        elif op == "graph_wide":
            c.update(queries=_between(rng, 2, 8000), tuning=rng.choice(["default", "latency"] + (
                [] if c["data"] == "unit" else ["throughput"])), host=rng.random() < 0.5)
        return c
    if op in ("linear_one", "linear_tc"):
        c = {"op": op, "data": rng.choice(["clusters", "bytes", "unit"]), "rows": _between(rng, 20_000, 700_000),
             "dim": _between(rng, 32, 960), "queries": 1, "k": _between(rng, 1, 200)}
        if op == "linear_tc":
            c.update(queries=_between(rng, 1, 8000), candidates=rng.choice([0, 256, 400]), ties=rng.random() < 0.5,
                     host=rng.random() < 0.5)
        return c
    if op in ("qg_exact", "qg_relaxed"):
        return {"op": op, "data": "bytes", "rows": _between(rng, 20_000, 200_000), "dim": 16 * rng.randint(3, 10),
                "queries": _between(rng, 1, 8000), "k": _between(rng, 1, 50), "epsilon": round(rng.uniform(0, 0.05), 3),
                "expansion": float(rng.choice([1, 3, 10]))}
    return {"op": op, "data": "bytes", "rows": _between(rng, 50_000, 1_000_000), "dim": 16 * rng.randint(3, 10),
            "queries": _between(rng, 1, 3000), "k": _between(rng, 1, 20), "probes": _between(rng, 4, 64),
            "expansion": float(rng.choice([3, 10])), "two_step": rng.random() < 0.7}


# ---- data -------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _points(data, n, dim, seed):
    """n float32 rows on the GPU: seed 1 gives an index's objects, other seeds queries."""
    g = _generator(1000 + seed)
    if data == "exponential":
        return torch.empty((n, dim), device="cuda").exponential_(1.0 / 25.0, generator=g).round_().clamp_(max=255.0)
    if data == "bytes":                                    # rank 16, as the benchmark's low-rank bytes
        a = 10.0 * torch.randn((16, dim), device="cuda", generator=_generator(7))
        z = torch.randn((n, 16), device="cuda", generator=g)
        return _spread(z, a).add_(128.0).round_().clamp_(0.0, 255.0)
    if data == "unit":                                     # rank 24 and some noise, unit length
        a = torch.randn((24, dim), device="cuda", generator=_generator(8))
        z = torch.randn((n, 24), device="cuda", generator=g)
        x = _spread(z, a).add_(torch.randn((n, dim), device="cuda", generator=g))
        return x / x.norm(dim=1, keepdim=True)
    means = torch.randn((64, dim), device="cuda", generator=_generator(9))
    x = means[torch.randint(0, 64, (n,), device="cuda", generator=g)]
    x += 0.5 * torch.randn((n, dim), device="cuda", generator=g)
    return x / x.norm(dim=1, keepdim=True)


def _spread(z, a):
    """z @ a without the tensor cores' rounding and in one order of summation."""
    out = torch.zeros((z.shape[0], a.shape[1]), device=z.device)
    for j in range(z.shape[1]):
        out.addcmul_(z[:, j:j + 1], a[j:j + 1])
    return out


DISTANCE = {"exponential": "L2", "bytes": "L2", "unit": "Cosine", "clusters": "NormalizedCosine"}


# ---- indexes in NGT's on-disk format -------------------------------------------------------

def _nearest(x, k):
    """The k nearest other rows of every row of x: ids (1-based) and L2 distances."""
    n = x.shape[0]
    before = torch.backends.cuda.matmul.allow_tf32
    # TF32 products of whole numbers up to 255 are exact, and so are their fp32 sums
    torch.backends.cuda.matmul.allow_tf32 = bool((x == x.round()).all())
    try:
        sq, xt = (x * x).sum(1), x.T.contiguous()
        ids = torch.empty((n, k), dtype=torch.int64, device="cuda")
        dst = torch.empty((n, k), device="cuda")
        step = max(128, min(4096, (1 << 30) // n))
        for s in range(0, n, step):
            e = min(n, s + step)
            d = torch.addmm(sq, x[s:e], xt, alpha=-2.0)
            d[torch.arange(e - s, device="cuda"), torch.arange(s, e, device="cuda")] = float("inf")
            v, i = torch.topk(d, k, dim=1, largest=False, sorted=True)
            ids[s:e], dst[s:e] = i + 1, (v + sq[s:e, None]).clamp_min(0).sqrt()
        return ids, dst
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before


def _graph(x, k=60, outgoing=10):
    """Each row's `outgoing` nearest and the rows that have it among their k nearest, by
    distance: counts per row, neighbour ids and distances, row after row."""
    n = x.shape[0]
    ids, dst = _nearest(x, k)
    own = torch.arange(1, n + 1, device="cuda")[:, None]
    src = torch.cat([own.expand(n, outgoing).reshape(-1), ids.reshape(-1)])
    to = torch.cat([ids[:, :outgoing].reshape(-1), own.expand(n, k).reshape(-1)])
    dd = torch.cat([dst[:, :outgoing].reshape(-1), dst.reshape(-1)])
    o = torch.argsort((src << 32) | to, stable=True)       # the copies of an edge beside each other
    src, to, dd = src[o], to[o], dd[o]
    keep = torch.ones_like(src, dtype=torch.bool)
    keep[1:] = (src[1:] != src[:-1]) | (to[1:] != to[:-1])
    src, to, dd = src[keep], to[keep], dd[keep]
    o = torch.argsort((src << 32) | dd.view(torch.int32).long(), stable=True)
    src, to, dd = src[o], to[o], dd[o]
    return torch.bincount(src - 1, minlength=n), to, dd


def _write_index(path, x, graph, distance):
    """A graph-only float index: prf, obj and grp of objects 1..n."""
    n, dim = x.shape
    os.makedirs(path)
    prf = {"Dimension": dim, "DistanceType": distance, "ObjectType": "Float-4", "IndexType": "Graph",
           "GraphType": "ONNG", "EdgeSizeForSearch": -2, "EdgeSizeForCreation": 100, "SeedSize": 10,
           "SeedType": "None", "EpsilonType": "None", "DynamicEdgeSizeBase": 30, "DynamicEdgeSizeRate": 20,
           "DatabaseType": "Memory", "ObjectAlignment": "False", "RefinementObjectType": "Float-4",
           "OutgoingEdge": 10, "IncomingEdge": 100}
    with open(os.path.join(path, "prf"), "w") as f:
        f.write("".join("%s\t%s\n" % kv for kv in sorted(prf.items())))
    head = struct.pack("<Q", n + 1) + b"-"
    with open(os.path.join(path, "obj"), "wb") as f:
        f.write(head)
        for s in range(0, n, 1 << 18):
            raw = x[s:s + (1 << 18)].contiguous().view(torch.uint8)
            mark = torch.full((raw.shape[0], 1), ord("+"), dtype=torch.uint8, device="cuda")
            torch.cat([mark, raw], 1).cpu().numpy().tofile(f)
    count, to, dd = graph
    start = torch.cumsum(5 + 8 * count, 0) - (5 + 8 * count)
    buf = torch.empty(int((5 + 8 * count).sum()), dtype=torch.uint8, device="cuda")
    buf[start] = ord("+")
    cb = count.int().view(-1, 1).view(torch.uint8)
    for t in range(4):
        buf[start + 1 + t] = cb[:, t].contiguous()
    first = torch.cumsum(count, 0) - count
    rank = torch.arange(len(to), device="cuda") - torch.repeat_interleave(first, count)
    at = torch.repeat_interleave(start, count) + 5 + 8 * rank
    pair = torch.stack([to.int(), dd.float().view(torch.int32)], 1).view(torch.uint8)
    for t in range(8):
        buf[at + t] = pair[:, t].contiguous()
    with open(os.path.join(path, "grp"), "wb") as f:
        f.write(head)
        buf.cpu().numpy().tofile(f)
        f.write(struct.pack("<I", n + 1) + bytes(2 * (n + 1)))


def _ring(n):
    """A graph that no case searches: every row's one edge leads to the next."""
    one = torch.ones(n, dtype=torch.int64, device="cuda")
    return one, torch.arange(1, n + 1, device="cuda") % n + 1, torch.zeros(n, device="cuda")


def _write_blobs(path, x, nblobs, nsid=64, dsv=2):
    """A quantized-blob-graph index of the byte rows x: blobs around means of the rows
    nearest to sampled rows, a random rotation, 16 centroids per subspace.  Sums are over
    whole numbers or run on the host in one order, so that every build is the same."""
    n, d = x.shape
    m = d // dsv
    rng = np.random.default_rng(5)
    x = x.double()

    def assign(c):
        norm = (c * c).sum(1)
        return torch.cat([(norm - 2.0 * (x[s:s + 8192] @ c.T)).argmin(1) for s in range(0, n, 8192)])

    blobs = x[torch.from_numpy(rng.choice(n, nblobs, replace=False)).cuda()]
    for _ in range(2):
        blob = assign(blobs)
        cnt = torch.bincount(blob, minlength=nblobs)
        total = torch.zeros_like(blobs).index_add_(0, blob, x)
        blobs = torch.where(cnt[:, None] > 0, total / cnt.clamp_min(1)[:, None], blobs).float().double()
    blob = assign(blobs)
    means = blobs[torch.from_numpy(rng.choice(nblobs, nsid, replace=False)).cuda()]
    norm = (means * means).sum(1)
    sid = (norm - 2.0 * (blobs @ means.T)).argmin(1)
    rot = torch.from_numpy(np.linalg.qr(rng.standard_normal((d, d)))[0]).cuda().float().double()
    rotated = (means @ rot).float().double()
    pick = torch.from_numpy(rng.choice(n, min(n, 16384), replace=False)).cuda()
    res = (x[pick] @ rot - rotated[sid[blob[pick]]]).cpu().numpy().reshape(-1, m, dsv)
    local = res[:16].transpose(1, 0, 2).copy()             # m, 16, dsv
    for _ in range(6):
        a = np.argmin([((res - local[None, :, c]) ** 2).sum(2) for c in range(16)], 0) + 16 * np.arange(m)
        cnt = np.bincount(a.ravel(), minlength=16 * m).reshape(m, 16)
        for j in range(dsv):
            s = np.bincount(a.ravel(), weights=res[:, :, j].ravel(), minlength=16 * m).reshape(m, 16)
            local[:, :, j] = np.where(cnt > 0, s / np.maximum(cnt, 1), local[:, :, j])
    lc = torch.from_numpy(local).cuda().float().double()
    codes = torch.empty((n, m), dtype=torch.uint8, device="cuda")
    for s in range(0, n, 16384):
        r = (x[s:s + 16384] @ rot - rotated[sid[blob[s:s + 16384]]]).view(-1, m, 1, dsv)
        codes[s:s + 16384] = ((r - lc) ** 2).sum(3).argmin(2).to(torch.uint8)
    _write_index(os.path.join(path, "global"), blobs.float(), _graph(blobs.float()), "L2")
    order = torch.argsort(blob, stable=True).cpu().numpy()
    cnt = torch.bincount(blob, minlength=nblobs).cpu().numpy()
    codes, sid = codes.cpu().numpy(), sid.cpu().numpy()
    with open(os.path.join(path, "grp"), "wb") as f:
        f.write(struct.pack("<QQII", m, nblobs + 1, 0, 0))
        at = 0
        for b in range(nblobs):
            mine = order[at:at + cnt[b]]
            at += cnt[b]
            f.write(struct.pack("<II", int(sid[b]), len(mine)))
            f.write((mine + 1).astype(np.uint32).tobytes())
            c = np.zeros(((len(mine) + 15) // 16 * 16, (m + 1) // 2 * 2), np.uint8)
            c[:len(mine), :m] = codes[mine]
            c = c.reshape(-1, 16, c.shape[1]).transpose(0, 2, 1)
            f.write((c[:, :, 0::2] | (c[:, :, 1::2] << 4)).tobytes())
    with open(os.path.join(path, "qr"), "wb") as f:
        f.write(struct.pack("<I", d * d) + rot.float().cpu().numpy().tobytes())
    with open(os.path.join(path, "rqcb"), "wb") as f:
        f.write(struct.pack("<III", nsid * d, d, d) + rotated.float().cpu().numpy().tobytes())
    for s in range(m):
        os.makedirs(os.path.join(path, "local-%d" % s))
        qg_build.write_object_file(os.path.join(path, "local-%d" % s, "obj"), lc[s].float().cpu().numpy())
    with open(os.path.join(path, "prf"), "w") as f:
        for kv in (("Dimension", d), ("GenuineDimension", d), ("LocalDivisionNo", m), ("LocalCentroidLimit", 16),
                   ("GlobalCentroidLimit", nsid), ("SingleLocalCodebook", 0), ("DistanceType", 1), ("DataType", 1),
                   ("GenuineDataType", 0), ("QuantizerType", 2)):
            f.write("%s\t%s\n" % kv)
    with open(os.path.join(path, "obj"), "wb") as f:
        f.write(struct.pack("<QQ", d, 0) + bytes(16 + d))
        rec = np.zeros((n, 16 + d), np.uint8)
        rec[:, 16:] = x.to(torch.uint8).cpu().numpy()
        rec.tofile(f)


def _kind(case):
    return case["op"].split("_")[0]                        # graph, linear, qg or qbg


def _index_path(case):
    """The case's index, built the first time and kept for later processes."""
    root = os.path.join(tempfile.gettempdir(), "ngt_cases_%d" % os.getuid())
    kind = _kind(case)
    path = os.path.join(root, "%s_%s_%d_%d" % (kind, case["data"], case["rows"], case["dim"]))
    if os.path.isdir(path):
        return path
    os.makedirs(root, exist_ok=True)
    work = tempfile.mkdtemp(dir=root)
    x = _points(case["data"], case["rows"], case["dim"], 1)
    made = os.path.join(work, "index")
    if kind == "qbg":
        _write_blobs(made, x, nblobs=max(256, case["rows"] // 128))
    else:
        _write_index(made, x, _ring(len(x)) if kind == "linear" else _graph(x), DISTANCE[case["data"]])
        if kind == "qg":
            qg_build.build_qg(made, x.cpu().numpy(), dsv=1, max_edges=64, log=lambda *a: None)
    del x
    torch.cuda.empty_cache()
    try:
        os.rename(made, path)
    except OSError:                                        # another process was faster
        pass
    shutil.rmtree(work, ignore_errors=True)
    return path


_open = {}


def _handle(case):
    """The open index that a program keeps; settings belong to the handle."""
    tuning = case.get("tuning", "default")
    key = (_index_path(case), tuning)
    if key not in _open:
        kind = _kind(case)
        if kind == "qg":
            ix = QuantizedIndex(key[0], zero_based_numbering=False)
        elif kind == "qbg":
            ix = QBGIndex(key[0])
        else:
            ix = Index(key[0], read_only=True)
            if tuning != "default":
                ix.set_batched_tuning(**TUNINGS[tuning])
        _open[key] = ix
    return _open[key]


# ---- the cases ------------------------------------------------------------------------------

class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.ix = case, _handle(case)
    q = _points(case["data"], case["queries"], case["dim"], 2 + seed).cpu().numpy()
    s.nq, s.k, s.queries = case["queries"], case["k"], q
    op = case["op"]
    if op in ("graph_wide", "linear_tc") and not case["host"] or op in ("qg_relaxed", "qbg"):
        if op == "qbg":
            rows = np.zeros((s.nq, s.ix._lib.ngtgpu_query_row_bytes(s.ix._index, s.ix._err)), np.uint8)
            s.ix._check(s.ix._lib.ngtgpu_convert_queries_float(s.ix._index, q.ctypes.data, s.nq, q.shape[1],
                                                               rows.ctypes.data, s.ix._err))
        else:
            rows = s.ix.convert_queries(q)
        s.rows = torch.from_numpy(rows).cuda()
        s.width = s.k
        if op == "qbg":
            s.flags = QBG_REFINE | (QBG_TWO_STEP if case["two_step"] else 0)
            s.params = QBGIndex.params(s.k, 0.1, 0.0, case["expansion"], case["probes"], 0)
        elif op == "qg_relaxed":
            s.params = QGQueryParameters(s.k, case["epsilon"], case["expansion"], -1.0)
        elif op == "graph_wide":
            s.params, s.nparams = Index.make_params(s.k, case["epsilon"])
        s.found = torch.zeros((s.nq, s.width, 2), dtype=torch.int32, device="cuda")
        s.counts = torch.zeros(s.nq, dtype=torch.int32, device="cuda")
        s.stats = torch.zeros((s.nq, 5), dtype=torch.int32, device="cuda")
        s.status = torch.zeros(s.nq, dtype=torch.int32, device="cuda")
    return s


def run(s):
    c, ix = s.case, s.ix
    op = c["op"]
    if op in ("graph_one", "linear_one"):
        got = ix.search(s.queries[0], k=s.k, epsilon=c["epsilon"]) if op == "graph_one" else \
            ix.linear_search(s.queries[0], k=s.k)
        return {"ids": np.array([r.id for r in got], np.uint32),
                "distances": np.array([r.distance for r in got], np.float32)}
    if op == "linear_tc" and c["host"]:
        ids, distances, counts, status = ix.linear_search_tc(s.queries, k=s.k, candidates=c["candidates"],
                                                             fp64_ties=c["ties"])
        return {"ids": ids, "distances": distances, "counts": counts, "status": status}
    if op == "graph_exact" or op == "graph_wide" and c["host"]:
        ids, distances, counts = ix.batch_search(s.queries, k=s.k, epsilon=c["epsilon"],
                                                 kernel=KERNEL_EXACT if op == "graph_exact" else KERNEL_WIDE)
        return {"ids": ids, "distances": distances, "counts": counts}
    if op == "qg_exact":
        ids, distances, counts = ix.batch_search(s.queries, size=s.k, epsilon=c["epsilon"],
                                                 result_expansion=c["expansion"])
        return {"ids": ids, "distances": distances, "counts": counts}
    out = {"ids": s.found[:, :, 0], "distances": s.found[:, :, 1].view(torch.float32), "counts": s.counts}
    if op == "graph_wide":
        ix.search_device(s.rows.data_ptr(), s.nq, s.params, s.nparams, s.found.data_ptr(), s.k, s.counts.data_ptr(),
                         s.stats.data_ptr(), kernel=KERNEL_WIDE)
    elif op == "linear_tc":
        ix._check(ix._lib.ngtgpu_linear_search_tc_ex(ix._index, s.rows.data_ptr(), s.nq, s.k, c["candidates"], 0,
                                                     1 if c["ties"] else 0, s.found.data_ptr(), s.k,
                                                     s.counts.data_ptr(), s.status.data_ptr(), None, ix._err))
        out["status"] = s.status
    elif op == "qg_relaxed":
        ix.search_device(s.rows.data_ptr(), s.nq, s.params, s.found.data_ptr(), s.width, s.counts.data_ptr(),
                         s.stats.data_ptr(), kernel=KERNEL_WIDE)
    else:
        ix._check(ix._lib.qbg_gpu_search_batch_device(ix._index, s.rows.data_ptr(), s.nq, ctypes.byref(s.params), 1,
                                                      s.flags, s.found.data_ptr(), s.width, s.counts.data_ptr(),
                                                      s.stats.data_ptr(), None, ix._err))
    return out


def exact(case, seed):
    """The distances of the exhaustive searches in 64 bits.  A graph search's results
    depend on the walk, so there is no value for them without the walk itself."""
    if _kind(case) != "linear":
        return None
    x = _points(case["data"], case["rows"], case["dim"], 1)
    q = _points(case["data"], case["queries"], case["dim"], 2 + seed)
    k = min(case["k"], case["rows"])
    sq = (x * x).sum(1)
    out = torch.empty((case["queries"], k), dtype=torch.float64, device="cuda")
    few = min(case["rows"], k + 64)                        # the nearest in 32 bits and some more, then 64 bits
    for s in range(0, case["queries"], 256):
        qq = q[s:s + 256]
        near = torch.topk(torch.addmm(sq, qq, x.T, alpha=-2.0), few, dim=1, largest=False)[1]
        y, z = x[near].double(), qq.double()[:, None, :]
        if DISTANCE[case["data"]] == "L2":
            d = (y - z).square().sum(2).sqrt()
        else:
            dot, length = (y * z).sum(2), z.norm(dim=2)
            d = 1.0 - dot / length if DISTANCE[case["data"]] == "NormalizedCosine" else \
                1.0 - dot / (length * y.norm(dim=2))
        out[s:s + 256] = torch.sort(d.abs(), dim=1)[0][:, :k]
    if case["op"] == "linear_one":
        return {"ids": None, "distances": out[0].cpu().numpy()}
    got = {"ids": None, "distances": out, "counts": None, "status": None}
    return {n: v.cpu().numpy() if case["host"] and v is not None else v for n, v in got.items()}


def work(case):
    """Bytes and operations of one pass.  For the graph searches the rows compared per
    query are a fit to the library's own counters over these indexes (exact within about
    a factor of two); a row is read in the form its kernel searches."""
    n, d, nq, k = case["rows"], case["dim"], case["queries"], case["k"]
    io = nq * (4 * d + 8 * k)
    op = case["op"]
    if op == "linear_one":
        return {"bytes": 4 * n * d + io, "flops": 2 * n * d}
    if op == "linear_tc":
        return {"bytes": 2 * n * d + io, "flops": 2 * n * d * nq}
    if op == "qbg":
        scanned = nq * case["probes"] * 128
        return {"bytes": min(scanned, n) * (d / 4 + 4) + io + nq * k * case["expansion"] * d, "flops": scanned * d / 2}
    if op in ("qg_exact", "qg_relaxed"):
        wide = nq * min(n, 400 + 81 * k * max(1.0, case["expansion"]))
        return {"bytes": wide * (d / 2 + 4) + io + nq * k * case["expansion"] * 4 * d, "flops": wide * d}
    widen = {"exponential": 0.36 * d, "bytes": 10.0, "unit": 16.7}[case["data"]]
    seen = nq * min(0.5 * n, (400 + 15 * k) * math.exp(widen * case["epsilon"]))
    row = {"graph_wide": 1 if case["data"] != "unit" else 4}.get(op, 4) * d
    return {"bytes": seen * (row + 4) + io, "flops": 3 * seen * d}
