"""Performance cases of the Top-K SpMV engine: what its users have it do, from a tiny matrix and
one query to a few hundred queries on a few million rows.

A case is one resident matrix and one batch of queries.  A pass loads the queries, runs the
two-stage Top-K (or the FP32-only one) and has the results: through the host-buffer calls
(``Q_reset``, the call itself, ``read_topk``), the device-resident pair (``run_device``,
``finish``), the pre-quantised flow (``Q_reset_quantized``, the call, ``read_candidates``) or
``run_exact``.

Fields of a case:
  entry     "host", "device", "quantised" or "exact"
  rows, cols, degree, mean, cap   matrix shape; row degrees "uniform" in mean/2 .. 3 mean/2, all
            "fixed" at mean, or "gamma" (shape 2) with that mean, none above cap
  values    "uniform" in (0, 1), "abs" |N(0, 1)| or "normal" N(0, 1)
  bits, quant   4, 6 or 8; "sym" (one symmetric scale), "row" or "global" (unsigned)
  split, ck, k  row partitions of the candidate select, candidates kept, results returned
  queries, nq   "dense" U(0, 1), "signed" U(-1, 1) or "sparse" (5-30 % of the entries U(0, 1))
  graphs, tensor   the handle's FLAG_GRAPHS and FLAG_TENSOR
"""
import math

import numpy as np
import torch

from acceles_gb300 import engine as E

QUANT = {"sym": E.QUANT_SYM_GLOBAL, "row": E.QUANT_UNSIGNED_ROW, "global": E.QUANT_UNSIGNED_GLOBAL}


def _case(entry, rows, cols, bits, nq, name=None, degree="uniform", mean=20, cap=512,
          values="uniform", quant="sym", split=1, ck=1024, k=100, queries="dense", graphs=False,
          tensor=False):
    c = dict(entry=entry, rows=rows, cols=cols, degree=degree, mean=mean, cap=cap, values=values,
             bits=bits, quant=quant, split=split, ck=ck, k=k, queries=queries, nq=nq,
             graphs=graphs, tensor=tensor)
    if name:
        c["name"] = name
    return c


def listed():
    ref = dict(degree="fixed", values="abs", split=32, ck=512)  # the method's published defaults
    return [
        # a small catalogue and one query through the host calls: launches and latency only
        _case("host", 4096, 256, 8, 1, "tiny_host", ck=256, k=10),
        # the reference driver's own flow on its default configuration: a matrix and a query that
        # were quantised beforehand, one query, candidates read back
        _case("quantised", 400_000, 500, 6, 1, "reference_flow", **ref),
        # one query on a resident matrix larger than L2, replayed as a graph (latency-critical)
        _case("device", 10_000_000, 1024, 8, 1, "one_large", graphs=True),
        # a small serving batch with the default 6 bits and 32 partitions, host buffers
        _case("host", 1_000_000, 1024, 6, 8, "few_split", split=32, ck=512),
        # a handful of sparse queries on a ragged 4-bit matrix with per-row scales
        _case("device", 300_007, 777, 4, 5, "few_ragged", degree="gamma", mean=32, quant="row",
              queries="sparse", ck=256, k=50),
        # the default configuration's 100-query benchmark
        _case("host", 400_000, 500, 6, 100, "batch_default", graphs=True, **ref),
        # what a busy serving slot collects: some tens of queries, signed embedding-like data
        _case("device", 2_000_000, 1024, 8, 40, "batch_serving", values="normal",
              queries="signed", graphs=True),
        # the throughput workload: hundreds of queries on a large 8-bit matrix
        _case("device", 4_000_000, 1024, 8, 512, "batch_large", graphs=True),
        # 256 sparse queries on a skewed 4-bit matrix, tensor-core layout
        _case("device", 2_000_000, 1024, 4, 256, "tensor_sparse", degree="gamma", mean=32,
              quant="row", queries="sparse", ck=256, graphs=True, tensor=True),
        # less than one block of signed queries on a ragged 4-bit matrix, tensor-core layout
        _case("host", 500_001, 700, 4, 100, "tensor_ragged", values="normal", queries="signed",
              tensor=True),
        # FP32-only Top-K: the check of one query, and of the queries of a tuning or search step
        _case("exact", 400_000, 500, 6, 1, "exact_one", **ref),
        _case("exact", 1_000_000, 1024, 8, 16, "exact_batch"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    entry = rng.choice(["host", "host", "device", "device", "device", "quantised", "exact"])
    rows = _log(rng, 2000, 3_000_000)
    cols = rng.choice([1024, 500, rng.randint(96, 1024)])
    bits = rng.choice([4, 6, 8])
    quant = "sym" if entry == "quantised" else rng.choice(["sym", "sym", "row", "global"])
    signed = quant == "sym" and rng.random() < 0.4
    degree = rng.choice(["uniform", "uniform", "fixed", "gamma"])
    mean = rng.choice([20, 32, rng.randint(8, 40)])
    nq = _log(rng, 1, 32) if entry == "exact" else _log(rng, 1, 512)
    while nq * rows * mean > 512 * 4_000_000 * 20:
        nq = max(1, nq // 2)
    k = rng.choice([100, 10, rng.randint(1, 100)])
    split = rng.choice([1, 1, 32, rng.randint(2, 40)])
    ck = max(rng.choice([256, 512, 1024]), split)
    return _case(entry, rows, cols, bits, nq, degree=degree, mean=mean,
                 values="normal" if signed else rng.choice(["uniform", "abs"]), quant=quant,
                 split=split, ck=ck, k=k,
                 queries="signed" if signed else rng.choice(["dense", "sparse"]),
                 graphs=entry in ("host", "device") and rng.random() < 0.5,
                 tensor=bits == 4 and rng.random() < 0.5)


# ---- inputs ------------------------------------------------------------------------------------
def _inputs(c, seed):
    """The matrix as a CSR sorted by (row, col) and the queries, FP32, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rows, cols, mean = c["rows"], c["cols"], c["mean"]

    def rand(*n):
        return torch.rand(*n, device="cuda", generator=g)

    if c["degree"] == "gamma":  # shape 2: the sum of two exponentials
        d = (-(mean / 2) * (torch.log1p(-rand(rows)) + torch.log1p(-rand(rows)))).round()
    elif c["degree"] == "uniform":
        d = (mean // 2 + (rand(rows) * (2 * (mean - mean // 2) + 1))).floor()
    else:
        d = torch.full((rows,), float(mean), device="cuda")
    d = d.clamp(1, min(c["cap"], cols)).to(torch.int64)
    row = torch.repeat_interleave(torch.arange(rows, device="cuda"), d)
    col = torch.randint(0, cols, row.shape, device="cuda", generator=g)
    key = torch.unique(row * 1024 + col)  # a column drawn twice in a row is one entry
    row, col = key // 1024, key % 1024
    del key
    if c["values"] == "uniform":
        val = rand(row.shape[0])
    else:
        val = torch.randn(row.shape[0], device="cuda", generator=g)
        if c["values"] == "abs":
            val = val.abs_()
    ptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=rows), 0)
    q = rand(c["nq"], cols)
    if c["queries"] == "signed":
        q = q * 2 - 1
    elif c["queries"] == "sparse":
        keep = rand(c["nq"], cols) < 0.05 + 0.25 * rand(c["nq"], 1)
        keep[:, 0] = True
        q = q * keep
    return ptr, row, col, val, q


def _quantised(x, bits, signed, m):
    """quantify_matrix / quantify_vector: round half to even of M * (x / m), in float64."""
    big = ((1 << bits) - 1) // 2 if signed else (1 << bits) - 1
    y = torch.round(big * (x.double() / m))
    return y.clamp(-big - 1 if signed else 0, big)


def _quantised_queries(c, q):
    signed = c["quant"] == "sym"
    m = (q.abs() if signed else q).amax(1, keepdim=True).double()
    return _quantised(q, c["bits"], signed, m)


def prepare(case, seed):
    c = case
    ptr, row, col, val, q = _inputs(c, seed)
    flags = (E.FLAG_GRAPHS if c["graphs"] else 0) | (E.FLAG_TENSOR if c["tensor"] else 0)
    kw = dict(bits=c["bits"], quant=QUANT[c["quant"]], split=c["split"], ck=c["ck"],
              k_max=c["k"], max_batch=c["nq"], flags=flags)
    hcol = col.to(torch.int32).cpu().numpy().view(np.uint32)
    st = {"entry": c["entry"], "k": c["k"], "nq": c["nq"]}
    if c["entry"] == "quantised":
        qv = _quantised(val, c["bits"], True, val.abs().max().double()).to(torch.int8)
        hrow = row.to(torch.int32).cpu().numpy().view(np.uint32)
        st["eng"] = E.SpMV(c["rows"], c["cols"], row=hrow, col=hcol, qval=qv.cpu().numpy(), **kw)
        st["q"] = _quantised_queries(c, q).to(torch.int8).cpu().numpy()
        return st
    st["eng"] = E.SpMV(c["rows"], c["cols"], ptr=ptr.cpu().numpy().view(np.uint64), col=hcol,
                       val=val.cpu().numpy(), **kw)
    if c["entry"] == "device":
        st["q"] = q.contiguous()
        st["idx"] = torch.empty(c["nq"], c["k"], dtype=torch.int32, device="cuda")
        st["score"] = torch.empty(c["nq"], c["k"], dtype=torch.float32, device="cuda")
    else:
        st["q"] = q.cpu().numpy()
    return st


def run(state):
    eng, k, q = state["eng"], state["k"], state["q"]
    if state["entry"] == "device":
        eng.run_device(q.data_ptr(), state["nq"], k, state["idx"].data_ptr(),
                       state["score"].data_ptr())
        eng.finish()
        return state["idx"], state["score"]
    if state["entry"] == "quantised":
        eng.Q_reset_quantized(q)
        eng(k=k)
        idx, score = eng.read_topk()
        cand, cand_score, _ = eng.read_candidates(0)
        return idx.view(np.int32), score, cand.view(np.int32), cand_score
    eng.Q_reset(q)
    if state["entry"] == "exact":
        idx, score, _ = eng.run_exact(k=k)
    else:
        eng(k=k)
        idx, score = eng.read_topk()
    return idx.view(np.int32), score


# ---- what a pass cannot do without -------------------------------------------------------------
def work(case):
    """Bytes: every nonzero once in its stored form (a B-bit value and a 10-bit column with a row
    flag; FP32 value, 16-bit column and row pointers in the FP32-only pass), the FP32 rows of the
    candidates, the queries and the results.  Flops: a multiply and an add per nonzero and query."""
    c = case
    nnz = c["rows"] * c["mean"]
    q = c["nq"] * c["cols"] * (1 if c["entry"] == "quantised" else 4)
    out = c["nq"] * c["k"] * 8
    if c["entry"] == "exact":
        return {"bytes": nnz * 6 + c["rows"] * 4 + q + out, "flops": 2 * nnz * c["nq"]}
    rescored = 0 if c["entry"] == "quantised" else c["nq"] * min(c["ck"], c["rows"]) * c["mean"]
    scales = 4 * c["rows"] if c["quant"] == "row" else 0
    return {"bytes": nnz * (c["bits"] + 11) / 8 + scales + rescored * 6 + q + out,
            "flops": 2 * (nnz * c["nq"] + rescored)}


# ---- the same in 64 bits -----------------------------------------------------------------------
def exact(case, seed):
    """Scores in float64, laid out as run() returns them; row indexes have no such value."""
    c = case
    ptr, row, col, val, q = _inputs(c, seed)
    rows, k, nq = c["rows"], c["k"], c["nq"]
    if nq * row.shape[0] > 1e11:
        return None
    val64, q64 = val.double(), q.double()
    ids = torch.arange(rows, device="cuda")

    def sums(v, x):  # per row, the sum over its entries of v * x[col]
        s = torch.cumsum(v * x[col], 0)
        s = torch.cat([s.new_zeros(1), s])
        return s[ptr[1:]] - s[ptr[:-1]]

    if c["entry"] == "exact":
        top = [torch.sort(torch.topk(sums(val64, q64[i]), min(k, rows)).values,
                          descending=True).values for i in range(nq)]
        return None, torch.stack(top)

    bits, signed = c["bits"], c["quant"] == "sym"
    scale = None
    if c["quant"] == "row":
        m = torch.zeros(rows, device="cuda").scatter_reduce_(0, row, val, "amax").double()
        scale = (m / ((1 << bits) - 1)).float()
        qv = _quantised(val, bits, False, m[row])
    else:
        qv = _quantised(val, bits, signed, val.abs().max().double())
    qq = _quantised_queries(c, q)
    split = max(1, c["split"])
    size = rows // split
    part = [(p * size, rows if p == split - 1 else (p + 1) * size) for p in range(split)]
    per = c["ck"] // split
    score = []
    for i in range(nq):
        s = torch.round(sums(qv, qq[i]))  # sums of integers: exact
        rank = s.to(torch.int64)
        if scale is not None:
            rank = (s.float() * scale).view(torch.int32).to(torch.int64)
        rank = (rank << 32) + ids  # by key, then by row
        pick = torch.cat([torch.topk(rank[a:b], min(per, b - a)).indices + a for a, b in part])
        if c["entry"] == "quantised":
            final = s[pick]
        else:
            at = torch.repeat_interleave(pick, ptr[pick + 1] - ptr[pick])
            first = torch.cumsum(ptr[pick + 1] - ptr[pick], 0) - (ptr[pick + 1] - ptr[pick])
            slot = torch.repeat_interleave(torch.arange(pick.shape[0], device="cuda"),
                                           ptr[pick + 1] - ptr[pick])
            e = ptr[at] + torch.arange(at.shape[0], device="cuda") - first[slot]
            final = q64.new_zeros(pick.shape[0]).index_add_(0, slot, val64[e] * q64[i][col[e]])
        final = torch.sort(final, descending=True).values[:k]
        if final.shape[0] < k:  # fewer candidates than results: the rest is -inf
            final = torch.cat([final, final.new_full((k - final.shape[0],), -math.inf)])
        score.append(final)
    score = torch.stack(score)
    if c["entry"] == "quantised":
        return None, score, None, None
    return None, score
