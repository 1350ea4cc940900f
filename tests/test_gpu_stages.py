"""GPU parity of the stages around the candidate pass at the sizes where their forms change:
every result must equal the CPU oracle's (rows and FP32 scores bit for bit)."""
import numpy as np
import pytest

import oracle as orc
from acceles_gb300 import engine as E

pytestmark = pytest.mark.gpu


def _check(m, eng, Q, split, ck, k, every=1):
    eng.Q_reset(Q)
    eng(k=k)
    idx, sc = eng.read_topk()
    for i in range(0, Q.shape[0], every):
        oi, os_, cand = m.two_stage(Q[i], split, ck, k)
        n = len(oi)
        assert np.array_equal(idx[i, :n], oi), f"query {i}: rows"
        assert np.array_equal(sc[i, :n], os_), f"query {i}: scores"
        assert np.all(idx[i, n:] == 0xFFFFFFFF) and np.all(np.isneginf(sc[i, n:]))
        assert set(eng.read_candidates(i)[0].tolist()) == set(cand.tolist()), f"query {i}: candidates"


@pytest.mark.parametrize("nq,ck,k,deg,ties", [
    (1, 64, 64, 20, False),      # one CTA's rows exactly
    (1, 65, 3, 20, False),       # and one row more: two CTAs
    (2, 4096, 1024, 20, False),  # the most candidates and results
    (3, 1000, 257, 20, False),   # just past ranking by counting
    (3, 700, 256, 20, False),
    (1, 200, 90, 300, False),    # rows of more than one staged chunk, up to every column
    (320, 600, 40, 20, False),   # one CTA per query, groups of 32 rows
    (320, 150, 20, 150, False),  # one CTA per query, groups of 4 long rows
    (2, 2000, 100, 20, True),    # more equal scores than the selection's list holds
])
def test_final_forms(nq, ck, k, deg, ties):
    rows, cols = 6000, 1024
    ptr, col, val = E.gen_matrix(E.GEN_GAMMA_DEG if deg > 20 else E.GEN_UNIFORM_DEG, rows, cols,
                                 deg if deg > 20 else 10, 1024 if deg > 20 else 30, seed=7 + ck)
    rng = np.random.default_rng(ck)
    Q = (rng.random((nq, cols)) * 2 - 1).astype(np.float32)
    if ties:  # every row the same four entries
        ptr = np.arange(rows + 1, dtype=np.uint64) * 4
        col = np.tile(np.array([1, 5, 9, 13], np.uint32), rows)
        val = np.ones(4 * rows, np.float32)
    m = orc.Matrix(rows, cols, ptr, col, val, 8, 0)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k,
                 max_batch=nq)
    _check(m, eng, Q, 1, ck, k, every=max(1, nq // 4))


@pytest.mark.parametrize("rows,split,ck,stride,nq,deg", [
    (60000, 1, 512, 16, 2, 20),    # about 3.7k samples, rank up to 128: group maxima
    (60000, 1, 64, 16, 2, 20),     # a small rank: 128 groups of four threads
    (60000, 1, 2048, 4, 2, 20),    # a rank above 128: histograms
    (20000, 1, 256, 1, 2, 20),     # every row sampled
    (600, 1, 64, 1, 1, 20),        # a few more samples than a warp holds
    (500, 1, 64, 1, 1, 20),        # and as many as it does
    (60000, 32, 512, 4, 3, 20),    # a warp per (query, partition)
    (60000, 32, 512, 64, 3, 20),   # few samples: many survivors, past a warp's registers
    (60000, 7, 455, 16, 3, 20),    # 65 candidates per partition: a CTA each
    (30000, 2, 128, 2, 40, 20),    # 64 of them, batched pass
    (30000, 2, 128, 2, 400, 20),   # ... and a warp per pair for the select
    (60000, 32, 512, 64, 40, 20),  # a warp per pair, some pairs past its registers
    (30000, 1, 4096, 64, 2, 4),    # more survivors than the select keeps in registers
])
def test_threshold_and_select_forms(rows, split, ck, stride, nq, deg):
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, 512, max(1, deg // 2), deg, seed=rows + ck)
    Q = (np.random.default_rng(stride).random((nq, 512)) * 2 - 1).astype(np.float32)
    m = orc.Matrix(rows, 512, ptr, col, val, 8, 0)
    eng = E.SpMV(rows, 512, ptr=ptr, col=col, val=val, bits=8, split=split, ck=ck, k_max=50,
                 max_batch=nq, sample_stride=stride)
    _check(m, eng, Q, split, ck, 50, every=max(1, nq // 5))


@pytest.mark.parametrize("split,ck", [(1, 500), (1, 2000), (8, 400), (32, 512)])
def test_select_ties(split, ck):
    """Scores of a handful of values only: the boundary falls among thousands of equal keys and
    the larger rows stay."""
    rows, cols = 40000, 64
    rng = np.random.default_rng(split + ck)
    ptr = np.arange(rows + 1, dtype=np.uint64) * 2
    col = np.sort(rng.integers(0, 8, (rows, 2)) * 8 + np.array([0, 1]), axis=1).astype(np.uint32).reshape(-1)
    val = rng.integers(1, 3, 2 * rows).astype(np.float32)
    Q = np.ones((2, cols), np.float32)
    m = orc.Matrix(rows, cols, ptr, col, val, 6, 0)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=6, split=split, ck=ck, k_max=60, max_batch=2)
    _check(m, eng, Q, split, ck, 60)
    if split > 1:  # many pairs: a warp each
        Q = np.repeat(Q[:1], 100, axis=0)
        eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=6, split=split, ck=ck, k_max=60, max_batch=100)
        _check(m, eng, Q, split, ck, 60, every=33)


@pytest.mark.parametrize("bits,quant", [(4, 0), (4, 1), (4, 2), (6, 0), (6, 1), (6, 2), (8, 0), (8, 1), (8, 2)])
@pytest.mark.parametrize("rows,cols,lo,hi,split,nq", [
    (9, 40, 1, 6, 1, 2),            # less than a tile
    (20000, 1024, 10, 30, 1, 4),    # one group of four
    (30001, 777, 1, 4, 32, 7),      # several rows per span; two groups, the last short
    (3000, 500, 150, 400, 5, 5),    # rows over several packets and tiles; one query alone
    (20000, 333, 5, 12, 1500, 6),   # partitions of a few rows, thresholds in global memory
    (20000, 96, 8, 20, 3, 17),      # groups share the SMs; one query alone
])
def test_four_query_pass(bits, quant, rows, cols, lo, hi, split, nq):
    """A few queries per call (auto batch tile): four per matrix read, the last one alone where
    one is left over.  One query is all zero, another has a single entry."""
    ck = max(64, 2 * split) if split > 1 else 200
    k = 30
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, lo, hi, seed=rows + bits)
    if quant == 0:
        val = val * np.where(np.random.default_rng(1).random(val.shape[0]) < 0.5, -1, 1).astype(np.float32)
    rng = np.random.default_rng(nq)
    Q = rng.random((nq, cols)).astype(np.float32)
    if quant == 0:
        Q = Q * 2 - 1
    Q[1] = 0
    if nq > 2:
        Q[2] = 0
        Q[2, cols // 2] = 1
    m = orc.Matrix(rows, cols, ptr, col, val, bits, quant)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=bits, quant=quant, split=split, ck=ck,
                 k_max=k, max_batch=nq)
    _check(m, eng, Q, split, ck, k)


@pytest.mark.parametrize("rows,cols,kind,p0,p1,nq,k,ck,stride", [
    (30000, 1024, E.GEN_UNIFORM_DEG, 10, 30, 1, 100, 512, 0),   # one query: rows filtered as scored
    (30001, 1024, E.GEN_UNIFORM_DEG, 0, 30, 17, 100, 512, 0),   # a group of 16 and one; empty rows
    (30000, 333, E.GEN_UNIFORM_DEG, 10, 30, 12, 7, 512, 0),     # twelve in a group of 16
    (29999, 777, E.GEN_UNIFORM_DEG, 1, 3, 6, 33, 512, 0),       # six in a group of eight
    (6000, 1024, E.GEN_GAMMA_DEG, 200, 1024, 11, 20, 512, 0),   # rows longer than a staged chunk's share
    (9001, 100, E.GEN_UNIFORM_DEG, 0, 12, 4, 50, 128, 0),        # a lane per row; short and empty rows
    (9000, 200, E.GEN_UNIFORM_DEG, 20, 60, 3, 50, 128, 0),       # long chunks, by four and by eight
    (9000, 200, E.GEN_UNIFORM_DEG, 20, 60, 8, 50, 128, 0),
    (31, 64, E.GEN_UNIFORM_DEG, 1, 9, 3, 40, 64, 0),            # fewer rows than results: no sample
    (30000, 256, E.GEN_UNIFORM_DEG, 4, 9, 70, 100, 128, 256),   # four groups of 16 and six
])
def test_fp32_only_batches(rows, cols, kind, p0, p1, nq, k, ck, stride):
    ptr, col, val = E.gen_matrix(kind, rows, cols, p0, p1, seed=rows + nq)
    val = val - np.float32(0.4)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq,
                 sample_stride=stride)
    Q = (np.random.default_rng(nq).random((nq, cols)) * 2 - 1).astype(np.float32)
    allrows = np.arange(rows, dtype=np.uint32)
    eng.Q_reset(Q)
    for kk in (k, max(1, k // 2)):  # a second K re-plans the sample
        idx, sc, ns = eng.run_exact(k=kk)
        assert ns > 0
        for i in range(0, nq, max(1, nq // 6)):
            s = orc.rescore_f32(ptr, col, val, Q[i], allrows)
            ri, rs = orc.sort_tuples_f32(allrows, s)
            n = min(kk, rows)
            assert np.array_equal(idx[i, :n], ri[:n]) and np.array_equal(sc[i, :n], rs[:n]), i
            assert np.all(idx[i, n:] == 0xFFFFFFFF)


@pytest.mark.parametrize("rows,cols,quant,split,nq,ck,hot", [
    (4000, 1024, 0, 1, 200, 4000, 0),   # every score passes: the hit queues overflow
    (90000, 256, 0, 1, 130, 64, 300),   # rows that pass for every query, in one tile
    (90000, 256, 1, 4, 256, 64, 300),   # with row scales and partitions
    (5000, 100, 0, 1, 17, 64, 50),      # a launch of a column more than a warp's block
    (3000, 96, 1, 1, 25, 100, 40),      # one block of few queries
])
def test_tensor_hit_queues(rows, cols, quant, split, nq, ck, hot):
    """Hits of the tensor-core pass go through per-CTA queues: units with none, with bursts of one
    row for every query and with more hits than a queue holds give the oracle's candidates."""
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 4, 12, seed=rows)
    if hot:  # consecutive rows of many large entries
        d = np.diff(ptr).astype(np.int64)
        d[rows // 2:rows // 2 + hot] = cols // 2
        ptr = np.concatenate([[0], np.cumsum(d)]).astype(np.uint64)
        rng = np.random.default_rng(3)
        col = np.concatenate([np.sort(rng.choice(cols, n, replace=False)) for n in d]).astype(np.uint32)
        val = rng.random(int(ptr[-1])).astype(np.float32)
    m = orc.Matrix(rows, cols, ptr, col, val, 4, quant)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=4, quant=quant, split=split, ck=ck,
                 k_max=20, max_batch=nq, batch_tile=128, flags=E.FLAG_TENSOR)
    assert eng.info()["tensor_tiles"] == 1
    Q = np.random.default_rng(nq).random((nq, cols)).astype(np.float32)
    _check(m, eng, Q, split, ck, 20, every=max(1, nq // 6))


@pytest.mark.parametrize("rows,stride,nq,bits,quant", [
    (60000, 1, 40, 8, 0),     # every tile sampled, by fours of queries
    (90000, 1, 200, 6, 0),    # ... by blocks of 128 (tiles x groups above the rule's line)
    (40000, 8, 131, 4, 1),    # row scales; the last group of three
])
def test_sample_pass_forms(rows, stride, nq, bits, quant):
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, 600, 6, 18, seed=rows)
    m = orc.Matrix(rows, 600, ptr, col, val, bits, quant)
    eng = E.SpMV(rows, 600, ptr=ptr, col=col, val=val, bits=bits, quant=quant, split=1, ck=200, k_max=30,
                 max_batch=nq, batch_tile=128, sample_stride=stride)
    Q = np.random.default_rng(nq).random((nq, 600)).astype(np.float32)
    _check(m, eng, Q, 1, 200, 30, every=max(1, nq // 6))


def _filter_case(rows, cols, lo, hi, bits, quant, seed, signed):
    """A CSR with an empty row, a row of zeros and a row quantised to nothing, and its queries."""
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, lo, hi, seed=seed)
    d = np.diff(ptr).astype(np.int64)
    keep = np.ones(len(val), bool)
    e = rows // 3
    keep[int(ptr[e]):int(ptr[e + 1])] = False
    d[e] = 0
    col, val = col[keep], val[keep]
    ptr = np.concatenate([[0], np.cumsum(d)]).astype(np.uint64)
    val[int(ptr[5]):int(ptr[6])] = 0
    val[int(ptr[7]):int(ptr[8])] *= np.float32(1e-5)
    if signed:
        val = val * np.where(np.random.default_rng(seed).random(len(val)) < 0.5, -1, 1).astype(np.float32)
    return ptr, col, val


@pytest.mark.parametrize("bits,quant", [(4, 0), (4, 1), (4, 2), (6, 0), (6, 1), (6, 2), (8, 0), (8, 1), (8, 2)])
@pytest.mark.parametrize("rows,cols,lo,hi,split,nq,kind", [
    (40000, 1024, 10, 30, 1, 65, "dense"),    # one CTA's launch, the last block of one query
    (40001, 500, 5, 25, 32, 150, "dense"),    # a CTA pair; partitions
    (9000, 333, 100, 300, 3, 300, "mixed"),   # a pair and a single launch; rows of many pieces
    (130, 40, 2, 8, 1, 129, "mixed"),         # two row tiles
    (20000, 128, 5, 25, 2, 40, "dense"),      # part of a launch's columns
])
def test_filter_pass(bits, quant, rows, cols, lo, hi, split, nq, kind):
    """Batches of a handle for more than 64 queries without a memory limit: approximate FP8 scores filter
    the rows and an exact integer check follows; with a memory limit the dp4a pass runs.  Both give
    the oracle's candidates and Top-K."""
    ck, k = max(96, 3 * split), 25
    ptr, col, val = _filter_case(rows, cols, lo, hi, bits, quant, rows + bits, quant == 0)
    rng = np.random.default_rng(nq)
    Q = rng.random((nq, cols)).astype(np.float32)
    if quant == 0:
        Q = Q * 2 - 1
    if kind == "mixed":  # a zero query, one-sided ones and sparse ones beside the rest
        Q[1] = 0
        Q[2::3] = np.abs(Q[2::3])
        Q[3::5] *= rng.random((len(Q[3::5]), cols)) < 0.1
    m = orc.Matrix(rows, cols, ptr, col, val, bits, quant)
    kw = dict(ptr=ptr, col=col, val=val, bits=bits, quant=quant, split=split, ck=ck, k_max=k,
              max_batch=max(nq, 65), batch_tile=128)
    eng = E.SpMV(rows, cols, **kw)
    lim = E.SpMV(rows, cols, mem_limit=1 << 40, **kw)
    assert eng.info()["device_bytes"] > lim.info()["device_bytes"]
    for e in (eng, lim):
        _check(m, e, Q, split, ck, k, every=max(1, nq // 7))
        for i in (1, 2, 3):
            assert set(e.read_candidates(i)[0].tolist()) == set(m.two_stage(Q[i], split, ck, k)[2].tolist())
        # (only the zero query, whose rows all tie, may overflow its survivors)
        assert e.stats()["repaired"] <= (1 if kind == "mixed" else 0)
    # a view runs the same pass; a graph replays it
    v = eng.view(flags=E.FLAG_GRAPHS)
    for _ in range(2):
        _check(m, v, Q, split, ck, k, every=max(1, nq // 2))


def test_filter_pass_bounds_too_wide():
    """Scores closer together than the filter's bounds: nearly every row passes, the lists overflow,
    and the batch is run again (and later batches are run) with the dp4a pass; no query needs the
    slow path."""
    rows, cols, deg, nq, ck, k = 150_000, 512, 120, 70, 8, 8
    rng = np.random.default_rng(5)
    ptr = (np.arange(rows + 1) * deg).astype(np.uint64)
    start = rng.integers(0, cols - deg, rows)
    col = (start[:, None] + np.arange(deg)[None, :]).astype(np.uint32).reshape(-1)
    val = (115 + rng.integers(-1, 2, rows * deg)).astype(np.float32)
    val[0] = 127
    Q = (115 + rng.integers(-1, 2, (nq, cols))).astype(np.float32)
    Q[:, 0] = 127
    m = orc.Matrix(rows, cols, ptr, col, val, 8, 0)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq,
                 batch_tile=128, sample_stride=4, flags=E.FLAG_GRAPHS)
    for _ in range(2):
        _check(m, eng, Q, 1, ck, k, every=30)
    assert eng.stats()["repaired"] == 0


def test_filter_pass_not_for_repeated_columns():
    """A row holding a column twice would lose one value in the dense tile: the dp4a pass runs."""
    rows, cols, nq = 3000, 64, 70
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 3, 6, seed=2)
    r = np.repeat(np.arange(rows, dtype=np.uint32), np.diff(ptr).astype(np.int64))
    r = np.concatenate([r, np.array([9], np.uint32)])
    c = np.concatenate([col, col[int(ptr[9]):int(ptr[9]) + 1]])
    v = np.concatenate([val, np.array([0.9], np.float32)])
    kw = dict(row=r, col=c, val=v, bits=8, split=1, ck=64, k_max=10, max_batch=nq, batch_tile=128)
    eng, lim = E.SpMV(rows, cols, **kw), E.SpMV(rows, cols, mem_limit=1 << 40, **kw)
    Q = np.random.default_rng(1).random((nq, cols)).astype(np.float32)
    for e in (eng, lim):
        e.Q_reset(Q)
        e(k=10)
    assert np.array_equal(eng.read_topk()[0], lim.read_topk()[0])
    assert np.array_equal(eng.read_topk()[1], lim.read_topk()[1])
