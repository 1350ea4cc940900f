"""GPU tests of the tensor-core filter (6- and 8-bit batches) beside its forms: rows and values at
its edges, its memory, and how it gives way to the dp4a pass.  Results must equal the oracle's."""
import contextlib

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
        assert set(eng.read_candidates(i)[0].tolist()) == set(cand.tolist()), f"query {i}: candidates"


@pytest.mark.parametrize("bits,quant", [(8, 0), (6, 1), (8, 2)])
def test_rows_left_empty(bits, quant):
    """Rows that quantise to nothing score by one forced entry, at the place of their largest value:
    with rows of up to 90 entries that place belongs to any lane of the warp that quantises the row."""
    rows, cols, nq, ck, k = 5000, 512, 80, 300, 30
    rng = np.random.default_rng(bits)
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 33, 90, seed=bits)
    if quant == 1:  # per-row scales: only rows of zeros are left empty
        zero = np.repeat(rng.random(rows) < 0.7, np.diff(ptr).astype(np.int64))
        val[zero] = 0
    else:
        val *= np.float32(1e-4)
        val[3] = 1.0
    if quant == 0:
        val = val * np.where(rng.random(len(val)) < 0.5, -1, 1).astype(np.float32)
    Q = rng.random((nq, cols)).astype(np.float32)
    m = orc.Matrix(rows, cols, ptr, col, val, bits, quant)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=bits, quant=quant, split=1, ck=ck, k_max=k,
                 max_batch=nq, batch_tile=128)
    _check(m, eng, Q, 1, ck, k, every=9)


def _wide(rows=150_000, nq=70):
    """Rows and queries whose scores lie closer together than the filter's bounds."""
    cols, deg = 512, 120
    rng = np.random.default_rng(5)
    ptr = (np.arange(rows + 1) * deg).astype(np.uint64)
    start = rng.integers(0, cols - deg, rows)
    col = (start[:, None] + np.arange(deg)[None, :]).astype(np.uint32).reshape(-1)
    val = (115 + rng.integers(-1, 2, rows * deg)).astype(np.float32)
    val[0] = 127
    Q = (115 + rng.integers(-1, 2, (nq, cols))).astype(np.float32)
    Q[:, 0] = 127
    kw = dict(ptr=ptr, col=col, val=val, bits=8, split=1, ck=8, k_max=8, max_batch=nq, sample_stride=4)
    return rows, cols, Q, kw


def _launches(eng, Q, k):
    eng.Q_reset(Q)
    eng.stats(reset=True)
    ns = eng(k=k)
    return eng.stats(reset=True)["launches"], ns


@pytest.mark.parametrize("rows", [150_000, 600_000])
def test_ties_leave_the_filter_on(rows):
    """Queries of zeros tie every row: their survivors (and the filter's lists) overflow whatever the pass.
    The batch after such a one takes the filter again."""
    cols, nq, ck, k = 256, 80, 64, 20
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 4, 10, seed=rows)
    Q = np.random.default_rng(1).random((nq, cols)).astype(np.float32)
    Z = Q.copy()
    Z[::10] = 0
    m = orc.Matrix(rows, cols, ptr, col, val, 8, 0)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq)
    base, _ = _launches(eng, Q, k)
    _check(m, eng, Z, 1, ck, k, every=5)
    assert _launches(eng, Q, k)[0] == base
    _check(m, eng, Q, 1, ck, k, every=16)


def test_lists_that_overflow():
    """The batch is run again without the filter, the second run counts in its time, and a batch that
    is small enough for it takes the four-query pass while the filter rests."""
    rows, cols, Q, kw = _wide()
    eng, dp4a = E.SpMV(rows, cols, **kw), E.SpMV(rows, cols, mem_limit=1 << 40, **kw)
    assert eng.info()["device_bytes"] > dp4a.info()["device_bytes"] + 8 * 120 * rows  # it has the layout
    one, _ = _launches(dp4a, Q, 8)
    ns1 = min(_launches(dp4a, Q, 8)[1] for _ in range(3))
    two, ns2 = _launches(eng, Q, 8)
    assert two > one and eng.stats()["repaired"] == 0
    assert ns2 > ns1
    assert _launches(eng, Q, 8)[0] == two  # the second in a row; the filter rests for two batches
    four, _ = _launches(dp4a, Q[:40], 8)
    assert _launches(eng, Q[:40], 8)[0] == four
    assert _launches(eng, Q, 8)[0] == one
    assert _launches(eng, Q, 8)[0] == two
    m = orc.Matrix(rows, cols, kw["ptr"], kw["col"], kw["val"], 8, 0)
    for _ in range(2):
        _check(m, eng, Q, 1, 8, 8, every=30)


def test_lists_hold_every_row_twice():
    """80 queries: the second 32 are shared by two epilogue warps, which append the same rows to one list;
    where every row passes, the lists still hold them and the batch is not run again."""
    rows, cols, ck, k = 20000, 128, 4096, 20
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 4, 10, seed=3)
    Q = np.random.default_rng(1).random((100, cols)).astype(np.float32)
    m = orc.Matrix(rows, cols, ptr, col, val, 8, 0)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=100)
    base, _ = _launches(eng, Q, k)
    assert _launches(eng, Q[:80], k)[0] == base
    _check(m, eng, Q[:80], 1, ck, k, every=13)


@pytest.mark.parametrize("bits,quant,bad", [(8, 1, np.nan), (6, 0, np.nan), (8, 0, np.inf), (8, 1, np.inf)])
def test_not_for_values_that_are_not_finite(bits, quant, bad):
    """An infinite or NaN value leaves its row's (or the matrix's) integers to the packer alone: the
    candidates are those of the dp4a pass."""
    rows, cols, nq, ck, k = 4000, 300, 70, 64, 20
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 5, 15, seed=4)
    for r in range(0, rows, 5):
        val[int(ptr[r])] = bad
    kw = dict(ptr=ptr, col=col, val=val, bits=bits, quant=quant, split=1, ck=ck, k_max=k, max_batch=nq,
              batch_tile=128)
    Q = np.random.default_rng(2).random((nq, cols)).astype(np.float32)
    got = []
    for e in (E.SpMV(rows, cols, **kw), E.SpMV(rows, cols, mem_limit=1 << 40, **kw)):
        e.Q_reset(Q)
        e(k=k)
        got.append([e.read_topk()[0]] + [e.read_candidates(i)[:2] for i in range(0, nq, 9)])
    assert np.array_equal(got[0][0], got[1][0])
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@contextlib.contextmanager
def _memory_short(left):
    """Holds device memory so that about `left` bytes stay free."""
    import torch
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(max(0, (free - left) >> 21) << 21, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        hold.untyped_storage().resize_(0)
        torch.cuda.empty_cache()


def test_layout_is_given_back_where_memory_is_short():
    """A matrix that fits beside the others' own memory is accepted: the layouts that nobody is using make
    room, and their handles go on with the dp4a pass."""
    rows, cols, nq, ck, k = 3_000_000, 256, 80, 64, 20
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 15, 25, seed=8)
    Q = np.random.default_rng(1).random((nq, cols)).astype(np.float32)
    kw = dict(ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq)
    m = orc.Matrix(rows, cols, ptr, col, val, 8, 0)
    probe = E.SpMV(rows, cols, mem_limit=1 << 40, **kw)
    alone = probe.info()["device_bytes"]
    dp4a, _ = _launches(probe, Q, k)
    probe.close()
    first = E.SpMV(rows, cols, flags=E.FLAG_GRAPHS, **kw)
    layout = first.info()["device_bytes"] - alone
    assert layout > 8 * int(ptr[-1])
    other = first.view()
    for e in (first, other):
        _check(m, e, Q, 1, ck, k, every=40)
    with _memory_short(alone + (64 << 20) - layout // 2):
        second = E.SpMV(rows, cols, **kw)
        assert first.info()["device_bytes"] <= alone + layout - 8 * int(ptr[-1])
        for e in (first, other, second):
            _check(m, e, Q, 1, ck, k, every=40)
            assert _launches(e, Q, k)[0] == dp4a


def test_lean_buffers_where_memory_is_short():
    """A view (and a retune) whose full buffers do not fit is made with the buffers of a limited handle."""
    rows, cols, nq, ck, k = 400_000, 256, 80, 1024, 20
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 15, 25, seed=9)
    Q = np.random.default_rng(1).random((nq, cols)).astype(np.float32)
    m = orc.Matrix(rows, cols, ptr, col, val, 8, 0)
    base = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq)
    v = base.view()
    full = v.info()["device_bytes"]
    v.close()
    v = base.view(mem_limit=1 << 40)
    lean = v.info()["device_bytes"]
    v.close()
    assert full > lean + (20 << 20)
    small = base.view(max_batch=1)
    _check(m, base, Q, 1, ck, k, every=40)
    with _memory_short((64 << 20) + (full + lean) // 2):
        small.retune(max_batch=nq)
        assert small.info()["device_bytes"] == lean
        _check(m, small, Q, 1, ck, k, every=40)
        small.close()
        v = base.view()
        assert v.info()["device_bytes"] == lean
        _check(m, v, Q, 1, ck, k, every=40)


def test_memory_limit_at_a_retune_leaves_no_layout():
    rows, cols, nq = 100_000, 256, 80
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 15, 25, seed=10)
    kw = dict(ptr=ptr, col=col, val=val, bits=8, split=1, ck=64, k_max=10, max_batch=nq)
    eng, lim = E.SpMV(rows, cols, **kw), E.SpMV(rows, cols, mem_limit=1 << 40, **kw)
    need = lim.info()["device_bytes"]
    eng.retune(mem_limit=need + (1 << 20))
    assert eng.info()["device_bytes"] <= need + (1 << 20)


def test_denser_sampling_keeps_the_fixed_scratch():
    """Many partitions: a denser sample would take this handle past the scratch of aes_run_noalloc."""
    import torch
    rows, cols, split, k = 1_500_000, 64, 2000, 10
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 5, 10, seed=3)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=split, ck=split, k_max=k)
    q = np.random.default_rng(1).random(cols).astype(np.float32)
    dq = torch.from_numpy(q).cuda()
    oi = torch.empty(k, dtype=torch.int32, device="cuda")
    os_ = torch.empty(k, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    eng.run_noalloc(dq.data_ptr(), k, oi.data_ptr(), os_.data_ptr())
    eng.Q_reset(q)
    eng(k=k)
    idx, sc = eng.read_topk()
    assert np.array_equal(oi.cpu().numpy().view(np.uint32), idx[0])
    assert np.array_equal(os_.cpu().numpy(), sc[0])


@pytest.mark.parametrize("quant,split", [(2, 1), (1, 3), (0, 1)])
def test_full_rows_of_large_values(quant, split):
    """Rows with an entry in every column, values and queries near the largest of 8 bits: scores near 2^26
    a few parts in a thousand apart, where the FP32 accumulation of the filter rounds most."""
    rows, cols, nq, ck, k = 3000, 1024, 70, 96, 30
    rng = np.random.default_rng(quant)
    ptr = np.arange(rows + 1, dtype=np.uint64) * cols
    col = np.tile(np.arange(cols, dtype=np.uint32), rows)
    val = (0.9 + 0.1 * rng.random(rows * cols)).astype(np.float32)
    Q = (0.9 + 0.1 * rng.random((nq, cols))).astype(np.float32)
    Q[1::2] = rng.random((len(Q[1::2]), cols))
    if quant == 0:
        val *= np.where(rng.random(len(val)) < 0.2, -1, 1).astype(np.float32)
    m = orc.Matrix(rows, cols, ptr, col, val, 8, quant)
    kw = dict(ptr=ptr, col=col, val=val, bits=8, quant=quant, split=split, ck=ck, k_max=k, max_batch=nq)
    eng, lim = E.SpMV(rows, cols, **kw), E.SpMV(rows, cols, mem_limit=1 << 40, **kw)
    assert eng.info()["device_bytes"] > lim.info()["device_bytes"] + 8 * int(ptr[-1])
    _check(m, eng, Q, split, ck, k, every=7)
    lim.Q_reset(Q)
    lim(k=k)
    for a, b in zip(eng.read_topk(), lim.read_topk()):
        assert np.array_equal(a, b)
    for i in range(nq):
        for a, b in zip(eng.read_candidates(i), lim.read_candidates(i)):
            assert np.array_equal(a, b)


def test_no_layout_where_a_row_repeats_a_column():
    """A large value given several times in one column: the dense tile would hold one of them, and the row, a
    candidate of every query, could be lost.  No layout is built, and blocks take the dp4a pass."""
    rows, cols, nq, ck, k = 3000, 64, 70, 64, 10
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 3, 6, seed=2)
    r = np.repeat(np.arange(rows, dtype=np.uint32), np.diff(ptr).astype(np.int64))
    plain = dict(row=r, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq)
    dup = dict(plain, row=np.concatenate([r, np.full(8, 9, np.uint32)]),
               col=np.concatenate([col, np.repeat(col[int(ptr[9])], 8)]),
               val=np.concatenate([val, np.full(8, 0.99, np.float32)]))
    Q = (0.5 + 0.5 * np.random.default_rng(1).random((nq, cols))).astype(np.float32)
    got = {}
    for name, kw in (("plain", plain), ("dup", dup), ("limit", dict(dup, mem_limit=1 << 40))):
        e = E.SpMV(rows, cols, **kw)
        e.Q_reset(Q)
        e(k=k)
        got[name] = (e.last_pass(), e.info()["device_bytes"], e.read_topk()[0])
    assert got["plain"][0] == E.PASS_FILTER and got["dup"][0] == got["limit"][0] == E.PASS_DP4A
    assert got["dup"][1] + 8 * len(val) < got["plain"][1]
    assert np.array_equal(got["dup"][2], got["limit"][2])
    assert all(9 in row for row in got["dup"][2])


def test_the_pass_that_gave_the_results():
    """Where the lists overflowed, the results are the dp4a pass's."""
    rows, cols, Q, kw = _wide()
    eng = E.SpMV(rows, cols, batch_tile=128, flags=E.FLAG_GRAPHS, **kw)
    eng.Q_reset(Q)
    eng(k=8)
    assert eng.last_pass() == E.PASS_DP4A


def test_layout_in_use_is_given_back_between_batches():
    """Threads that keep batches on a layout do not keep its memory from a create that needs it."""
    import threading
    rows, cols, nq, ck, k = 3_000_000, 256, 80, 64, 20
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 15, 25, seed=8)
    Q = np.random.default_rng(1).random((nq, cols)).astype(np.float32)
    kw = dict(ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq)
    probe = E.SpMV(rows, cols, mem_limit=1 << 40, **kw)
    alone = probe.info()["device_bytes"]
    probe.Q_reset(Q)
    probe(k=k)
    want = probe.read_topk()
    probe.close()
    first = E.SpMV(rows, cols, **kw)
    layout = first.info()["device_bytes"] - alone
    handles = [first, first.view(), first.view(flags=E.FLAG_GRAPHS)]
    seen, bad, stop = [set(), set(), set()], [], threading.Event()

    def serve(i):
        e = handles[i]
        while not stop.is_set():
            e.Q_reset(Q)
            e(k=k)
            seen[i].add(e.last_pass())
            idx, sc = e.read_topk()
            if not (np.array_equal(idx, want[0]) and np.array_equal(sc, want[1])):
                bad.append(i)

    threads = [threading.Thread(target=serve, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    try:
        while not all(E.PASS_FILTER in s for s in seen):
            assert any(t.is_alive() for t in threads)
        with _memory_short(alone + (64 << 20) - layout // 2):
            second = E.SpMV(rows, cols, **kw)
            second.Q_reset(Q)
            second(k=k)
            assert np.array_equal(second.read_topk()[0], want[0])
            for s in seen:
                s.clear()
            while not all(seen):
                assert any(t.is_alive() for t in threads)
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not bad
    assert all(s == {E.PASS_DP4A} for s in seen)


def test_layout_of_a_captured_batch_is_kept():
    """A caller's graph holds the layout's addresses: its replays stay valid, a create that would need that
    memory is refused."""
    import torch
    rows, cols, nq, ck, k = 3_000_000, 256, 80, 64, 20
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 15, 25, seed=8)
    rng = np.random.default_rng(1)
    Q = rng.random((2, nq, cols)).astype(np.float32)
    kw = dict(ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq)
    eng = E.SpMV(rows, cols, **kw)
    lim = E.SpMV(rows, cols, mem_limit=1 << 40, **kw)
    alone = lim.info()["device_bytes"]
    layout = eng.info()["device_bytes"] - alone
    want = []
    for q in Q:
        lim.Q_reset(q)
        lim(k=k)
        want.append(tuple(x.copy() for x in lim.read_topk()))
    lim.close()
    dq = torch.from_numpy(Q[0]).cuda()
    oi = torch.zeros((nq, k), dtype=torch.int32, device="cuda")
    os_ = torch.zeros((nq, k), dtype=torch.float32, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    eng.run_device(dq.data_ptr(), nq, k, oi.data_ptr(), os_.data_ptr(), s.cuda_stream)
    eng.finish()
    assert eng.last_pass() == E.PASS_FILTER
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        eng.run_device(dq.data_ptr(), nq, k, oi.data_ptr(), os_.data_ptr(), s.cuda_stream)

    def replay(i):
        dq.copy_(torch.from_numpy(Q[i]))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert eng.finish() == 0
        assert np.array_equal(oi.cpu().numpy().view(np.uint32), want[i][0])
        assert np.array_equal(os_.cpu().numpy(), want[i][1])

    replay(0)
    replay(1)
    with _memory_short(alone + (64 << 20) - layout // 2):
        with pytest.raises(E.AesError) as ei:
            E.SpMV(rows, cols, **kw)
        assert ei.value.code == E.AES_ERR_NOMEM
        replay(0)
    replay(1)
