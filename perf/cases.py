"""Cases that the framework's speed is measured on.

Each case is a call (or the short run of calls) that a program using the
library makes on a resident table: single scans, BinDex queries and builds,
batches of a few to a thousand queries, the host-buffer batch, the steps
after a scan (row ids, aggregates) and a served burst.  Column kinds are the
benchmark's and the tests' (uniform over 2^32, small domains, zipf over 2^20
values, a rounded normal); queries have log-uniform selectivity at random
centres, as the benchmark's.
"""
import math

import numpy as np
import torch

import rtscan_b200 as R
from rtscan_b200 import datagen as D

BATCH_KINDS = "zipf1.1,zipf1.3,zipf1.5,normal"
SERVE_KINDS = "uniform,uniform,zipf1.3,zipf1.3"
WIDE_KINDS = "uniform,zipf1.3,normal,uniform2p8,uniform,zipf1.1,uniform2p6,normal"
# TPC-H Q6, integer-coded: shipdate, discount, quantity, extended price
Q6_KINDS = "range:19920101:19990101,range:0:11,range:1:51,range:90000:10500000"
Q6_TERMS = [(0, 19940101, 19950100), (1, 5, 7), (2, 0, 23)]


def _case(name, op, rows, kinds, **more):
    c = {"name": name, "op": op, "rows": rows, "kinds": kinds, "nq": 1, "terms": 0, "min_sel": 1e-4, "max_sel": 0.9,
         "offset": 0}
    c.update(more)
    return c


def listed():
    return [
        # one predicate on a table of the size the tests use: a point lookup
        # in a small dimension table, where the launches are the cost
        _case("scan_small", "scan", 100_003, "uniform", terms=1),
        # an analytic filter over three columns of a mid-sized table
        _case("scan_3col", "scan", 30_000_001, "zipf1.3,normal,uniform", terms=3, min_sel=0.01),
        # two indexed columns at the reference's row count and area count
        _case("bindex_scan", "bindex", 100_000_000, "uniform,normal", terms=2, min_sel=0.01, max_sel=0.5),
        # building that index when a table is loaded, and its first query
        _case("bindex_build", "bindex_build", 1 << 25, "zipf1.3", terms=1, min_sel=0.01),
        # a handful of concurrent queries: what a lightly loaded server or a
        # dashboard's page sends at once
        _case("batch_16", "batch", 1 << 23, SERVE_KINDS, nq=16),
        # a dashboard's fixed set of queries, prepared once and replayed
        _case("batch_100_graph", "batch_graph", 20_000_003, SERVE_KINDS, nq=100),
        # many concurrent queries over a fact table with more columns than
        # the benchmark's, each query on one to four of them
        _case("batch_300_8col", "batch", 1 << 24, WIDE_KINDS, nq=300),
        # the benchmark's batched workload
        _case("batch_1024", "batch", 100_000_000, BATCH_KINDS, nq=1024),
        # columns in host memory, bitmaps wanted in host memory
        _case("batch_host", "batch_host", (1 << 23) + 77, "uniform,zipf1.3", nq=48),
        # TPC-H Q6: filter and sum in one pass
        _case("aggregate_q6", "aggregate", 60_000_000, Q6_KINDS, terms=3),
        # filter, then the row ids for late materialization
        _case("scan_rows", "rows", 1 << 25, "uniform,zipf1.3", terms=2, min_sel=0.1, max_sel=0.5),
        # a burst of requests at the server
        _case("served_burst", "served", 1 << 24, SERVE_KINDS, nq=200),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["scan", "scan", "bindex", "bindex_build", "batch", "batch", "batch", "batch_graph", "batch_host",
                     "aggregate", "rows", "served"])
    names = ["uniform", "uniform", "uniform2p6", "uniform2p8", "zipf1.1", "zipf1.3", "zipf1.5", "normal"]
    c = _case(None, op, 0, "")
    del c["name"]
    c["offset"] = rng.choice([0, 0, 0, 0, 1, 2])  # borrowed columns may start anywhere
    if op == "scan":
        k = rng.randint(1, 4)
        c.update(rows=_log_int(rng, 1_000, 100_000_000), terms=k)
    elif op == "bindex":
        k = rng.randint(1, 3)
        c.update(rows=_log_int(rng, 100_000, 100_000_000), terms=k, min_sel=1e-3)
    elif op == "bindex_build":
        k = 1
        c.update(rows=_log_int(rng, 100_000, 50_000_000), terms=1)
    elif op in ("batch", "batch_graph"):
        k = rng.randint(1, 8)
        nq = _log_int(rng, 2, 1024)
        most = max(20_000, min(100_000_000, 50_000_000_000 // nq // max(1, k // 4)))
        c.update(rows=_log_int(rng, 20_000, most), nq=nq)
    elif op == "batch_host":
        k = rng.randint(1, 4)
        nq = _log_int(rng, 2, 200)
        c.update(rows=_log_int(rng, 20_000, 8_000_000), nq=nq)
    elif op == "aggregate":
        k = 4
        c.update(rows=_log_int(rng, 10_000, 100_000_000), terms=3)
    elif op == "rows":
        k = rng.randint(1, 3)
        c.update(rows=_log_int(rng, 10_000, 100_000_000), terms=k, min_sel=1e-3)
    else:
        k = rng.randint(1, 6)
        c.update(rows=_log_int(rng, 200_000, 16_000_000), nq=_log_int(rng, 4, 300))
    c["kinds"] = Q6_KINDS if op == "aggregate" else ",".join(rng.choice(names) for _ in range(k))
    return c


def _column(kind, n, gen):
    """An int32 tensor holding the bits of n uint32 values."""
    dev = "cuda"
    if kind.startswith("range:"):
        _, lo, hi = kind.split(":")
        return torch.randint(int(lo), int(hi), (n,), generator=gen, device=dev, dtype=torch.int32)
    if kind == "uniform":
        return torch.randint(-(1 << 31), 1 << 31, (n,), generator=gen, device=dev, dtype=torch.int32)
    if kind.startswith("uniform2p"):
        return torch.randint(0, 1 << int(kind[9:]), (n,), generator=gen, device=dev, dtype=torch.int32)
    out = torch.empty(n, device=dev, dtype=torch.int32)
    step = 1 << 25
    if kind.startswith("zipf"):
        cdf = torch.cumsum(torch.arange(1, (1 << 20) + 1, device=dev, dtype=torch.float64) ** -float(kind[4:]), 0)
        cdf /= cdf[-1].clone()
        for a in range(0, n, step):
            u = torch.rand(min(step, n - a), generator=gen, device=dev, dtype=torch.float64)
            out[a:a + step] = torch.searchsorted(cdf, u, right=True).clamp_(max=(1 << 20) - 1).to(torch.int32)
        return out
    for a in range(0, n, step):  # normal, mean 2^31, sd 2^28: minus 2^31 as int32 has the bits of x - 2^32 or x
        z = torch.randn(min(step, n - a), generator=gen, device=dev, dtype=torch.float64)
        x = torch.round(z * 2.0 ** 28 + 2.0 ** 31).clamp_(0, 2.0 ** 32 - 1).to(torch.int64)
        out[a:a + step] = torch.where(x >= 1 << 31, x - (1 << 32), x).to(torch.int32)
    return out


def _table(case, seed):
    """The case's columns (views `offset` values into their storage) and
    its queries."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, off = case["rows"], case["offset"]
    cols = [_column(k, n + off, gen)[off:] for k in case["kinds"].split(",")]
    if case["op"] == "aggregate":
        return cols, [list(Q6_TERMS)]
    samples = []
    for c in cols:
        at = torch.randint(0, n, (min(n, 1 << 17),), generator=gen, device="cuda")
        samples.append(c[at].cpu().numpy().view(np.uint32))
    k = case["terms"]
    queries = D.batch_queries(samples, case["nq"], seed, case["min_sel"], case["max_sel"], min_cols=k or 1,
                              max_cols=k or 4)
    return cols, queries


class _State:
    """What a program holds: the context, its table and result buffers."""

    def __init__(self, case, seed):
        self.op = case["op"]
        self.cols, self.queries = _table(case, seed)
        self.terms = self.queries[0]
        n, nq = case["rows"], case["nq"]
        self.words = (n + 31) // 32
        self.stride = (self.words + 3) // 4 * 4
        self.ctx = R.Context(0)
        self.stream = torch.cuda.current_stream().cuda_stream
        if self.op == "batch_host":
            self.host_cols = [c.cpu().pin_memory().numpy().view(np.uint32) for c in self.cols]
            self.cols = None
            self.prepared = R.prepare(self.queries)
            self.host_bitmaps = torch.zeros((nq, self.stride), dtype=torch.int32).pin_memory().numpy().view(np.uint32)
            return
        self.ctx.attach_columns([c.data_ptr() for c in self.cols], n)
        if self.op == "served":
            self.server = R.Server(self.ctx, max_active=256, segment_rows=1 << 22)
            return
        if self.op == "aggregate":
            self.count = torch.zeros(1, dtype=torch.int64, device="cuda")
            self.sum = torch.zeros(2, dtype=torch.int64, device="cuda")
            return
        self.bitmaps = torch.zeros((nq, self.stride), dtype=torch.int32, device="cuda")
        self.counts = torch.zeros(nq, dtype=torch.int64, device="cuda")
        if self.op == "bindex":
            for c in sorted({t[0] for t in self.terms}):
                self.ctx.build_bindex(c, 128)
        elif self.op == "rows":
            self.rows = torch.zeros(n, dtype=torch.int32, device="cuda")
            self.nrows = torch.zeros(1, dtype=torch.int64, device="cuda")
        elif self.op in ("batch", "batch_graph"):
            self.prepared = R.prepare(self.queries)
            if self.op == "batch_graph":
                self.graph = self.ctx.prepare_batch(self.prepared, self.bitmaps.data_ptr(), self.stride,
                                                    self.counts.data_ptr())

    def __del__(self):
        for name in ("server", "graph"):
            h = getattr(self, name, None)
            if h is not None:
                h.stop() if name == "server" else h.release()


def prepare(case, seed):
    s = _State(case, seed)
    s.nrows_table = case["rows"]
    return s


def run(s):
    bm = s.bitmaps.data_ptr() if hasattr(s, "bitmaps") else 0
    cnt = s.counts.data_ptr() if hasattr(s, "counts") else 0
    if s.op == "scan":
        s.ctx.scan_async(s.terms, bm, cnt, s.stream)
        return [s.bitmaps, s.counts]
    if s.op == "bindex":
        s.ctx.bindex_scan_async(s.terms, bm, cnt, s.stream)
        return [s.bitmaps, s.counts]
    if s.op == "bindex_build":
        s.ctx.build_bindex(0, 128)
        s.ctx.bindex_scan_async(s.terms, bm, cnt, s.stream)
        starts, ranks = s.ctx.bindex_areas(0, 128)
        return [s.bitmaps, s.counts, starts.astype(np.int64), ranks.astype(np.int64)]
    if s.op == "batch":
        s.ctx.scan_batch_async(s.prepared, bm, s.stride, cnt, s.stream)
        return [s.bitmaps, s.counts]
    if s.op == "batch_graph":
        s.graph.launch(s.stream)
        return [s.bitmaps, s.counts]
    if s.op == "batch_host":
        out, counts = s.ctx.scan_batch_host(s.host_cols, s.prepared, s.host_bitmaps, s.stride)
        return [out.view(np.int32), counts.astype(np.int64)]
    if s.op == "aggregate":
        s.ctx.scan_aggregate_async(s.terms, 3, 1, s.count.data_ptr(), s.sum.data_ptr(), s.stream)
        return [s.count, s.sum]
    if s.op == "rows":
        s.ctx.scan_async(s.terms, bm, cnt, s.stream)
        s.ctx.bitmap_rows_async(bm, s.nrows_table, s.rows.data_ptr(), s.rows.numel(), s.nrows.data_ptr(), s.stream)
        return [s.bitmaps, s.counts, s.rows, s.nrows]
    tickets = [s.server.submit(q) for q in s.queries]
    counts = []
    for t in tickets:
        s.server.wait(t)
        counts.append(s.server.fetch(t, want_bitmap=False)[1])
    return np.array(counts, dtype=np.int64)


def work(case):
    n, nq = case["rows"], case["nq"]
    k = len(case["kinds"].split(","))
    op = case["op"]
    bitmap = n / 8
    if op == "bindex":  # up to two filter vectors per term, one result
        b = (2 * case["terms"] + 1) * bitmap
    elif op == "bindex_build":  # column in; sorted values, row ids and 127 filter vectors out
        b = 12 * n + 127 * bitmap
    elif op == "aggregate":
        b = 4 * n * k
    elif op == "rows":  # columns in, bitmap out and in, row ids of the smallest selectivity out
        b = 4 * n * case["terms"] + 2 * bitmap + 4 * n * case["min_sel"]
    elif op in ("batch", "batch_graph", "batch_host", "served"):
        b = 4 * n * (min(k, 4) if nq == 1 else k) + nq * bitmap
    else:
        b = 4 * n * case["terms"] + bitmap
    return {"bytes": float(b), "flops": 0.0}


def _mask(cols, terms, n):
    hit = torch.ones(n, dtype=torch.bool, device="cuda")
    for c, lo, hi in terms:
        x = cols[c].to(torch.int64) & 0xFFFFFFFF
        hit &= (x >= lo) & (x <= hi)
    return hit


def _pack(hit, stride):
    bits = torch.zeros(stride * 32, dtype=torch.int64, device="cuda")
    bits[:hit.numel()] = hit
    w = (bits.view(-1, 32) << torch.arange(31, -1, -1, device="cuda")).sum(1)
    return torch.where(w >= 1 << 31, w - (1 << 32), w).to(torch.int32)


def exact(case, seed):
    """The results as plain torch computes them (64-bit compares)."""
    n, nq, op = case["rows"], case["nq"], case["op"]
    if n * nq > 6_000_000_000:
        return None
    cols, queries = _table(case, seed)
    stride = (((n + 31) // 32) + 3) // 4 * 4
    if op == "served":
        return np.array([int(_mask(cols, q, n).sum()) for q in queries], dtype=np.int64)
    if op == "aggregate":
        hit = _mask(cols, queries[0], n)
        prod = (cols[3].to(torch.int64) * cols[1].to(torch.int64))[hit].sum()
        return [hit.sum().view(1), torch.stack([prod, torch.zeros_like(prod)])]
    bitmaps = torch.zeros((nq, stride), dtype=torch.int32, device="cuda")
    counts = torch.zeros(nq, dtype=torch.int64, device="cuda")
    for i, q in enumerate(queries):
        hit = _mask(cols, q, n)
        bitmaps[i] = _pack(hit, stride)
        counts[i] = hit.sum()
    if op == "rows":
        ids = torch.zeros(n, dtype=torch.int32, device="cuda")
        at = hit.nonzero().view(-1)
        ids[:at.numel()] = at.to(torch.int32)
        return [bitmaps, counts, ids, counts.clone()]
    if op == "bindex_build":
        x = torch.sort(cols[0].to(torch.int64) & 0xFFFFFFFF).values
        starts = x[torch.arange(128, device="cuda") * (n // 128)]
        return [bitmaps, counts, starts, torch.searchsorted(x, starts)]
    return [bitmaps, counts]
