"""GPU tests of calls that meet on one handle: a device-resident batch not yet finished and the
FP32-only pass, and that pass over more queries than there are SMs.  Results must equal the oracle's."""
import numpy as np
import pytest

import oracle as orc
from acceles_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [256, 255])  # 255: queries on the device are staged at a padded stride
def test_exact_pass_between_a_device_batch_and_its_finish(cols):
    """Queries of zeros tie every row and need the slow path; aes_finish still finds them after an
    aes_run_exact of other queries on the same handle."""
    import torch
    rows, nq, ck, k = 200_000, 5, 64, 20
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 4, 10, seed=cols)
    val = val - np.float32(0.5)
    rng = np.random.default_rng(1)
    Q = (rng.random((nq, cols)) * 2 - 1).astype(np.float32)
    Q[1::2] = 0
    X = (rng.random((nq, cols)) * 2 - 1).astype(np.float32)
    m = orc.Matrix(rows, cols, ptr, col, val, 8, 0)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=ck, k_max=k, max_batch=nq)
    eng.Q_reset(X)
    dq = torch.from_numpy(Q).cuda()
    oi = torch.zeros((nq, k), dtype=torch.int32, device="cuda")
    os_ = torch.zeros((nq, k), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    eng.run_device(dq.data_ptr(), nq, k, oi.data_ptr(), os_.data_ptr())
    xi, xs, _ = eng.run_exact(k=k)
    assert eng.finish() == 2
    torch.cuda.synchronize()
    allrows = np.arange(rows, dtype=np.uint32)
    for i in range(nq):
        ri, rs = orc.sort_tuples_f32(allrows, orc.rescore_f32(ptr, col, val, X[i], allrows))
        assert np.array_equal(xi[i], ri[:k]) and np.array_equal(xs[i], rs[:k]), f"exact {i}"
        ri, rs, _ = m.two_stage(Q[i], 1, ck, k)
        assert np.array_equal(oi[i].cpu().numpy().view(np.uint32), ri), f"device {i}"
        assert np.array_equal(os_[i].cpu().numpy(), rs), f"device {i}"
    assert eng.finish() == 0


def test_last_pass():
    rows, cols, k = 30_000, 256, 10
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 4, 10, seed=2)
    kw = dict(ptr=ptr, col=col, val=val, split=1, ck=64, k_max=k, max_batch=200)
    Q = np.random.default_rng(1).random((200, cols)).astype(np.float32)

    def passes(eng, *sizes):
        out = []
        for n in sizes:
            eng.Q_reset(Q[:n])
            eng(k=k)
            out.append(eng.last_pass())
        return out

    eng = E.SpMV(rows, cols, bits=8, flags=E.FLAG_GRAPHS, **kw)
    assert eng.last_pass() == E.PASS_NONE
    for _ in range(2):  # captured, replayed
        assert passes(eng, 1, 4, 32, 33, 100, 200) == [
            E.PASS_PLAIN, E.PASS_FOUR, E.PASS_FOUR, E.PASS_FILTER, E.PASS_FILTER, E.PASS_FILTER]
    eng.retune(batch_tile=1)
    assert passes(eng, 4, 100) == [E.PASS_PLAIN] * 2
    lim = E.SpMV(rows, cols, bits=8, mem_limit=1 << 40, **kw)
    assert passes(lim, 33, 48, 49, 200) == [E.PASS_FOUR, E.PASS_FOUR, E.PASS_DP4A, E.PASS_DP4A]
    ten = E.SpMV(rows, cols, bits=4, flags=E.FLAG_TENSOR, **kw)
    assert passes(ten, 12, 13, 200) == [E.PASS_FOUR, E.PASS_TENSOR, E.PASS_TENSOR]


@pytest.mark.parametrize("nq", [70, 128, 200])
def test_profile_covers_the_exact_check(nq):
    """The candidate pass's time of a filter launch holds its exact check: with wide bounds that check
    scores most rows for every query and takes longer than the FP8 products."""
    rows, cols, k = 60_000, 512, 10
    rng = np.random.default_rng(5)
    deg = 60
    ptr = (np.arange(rows + 1) * deg).astype(np.uint64)
    start = rng.integers(0, cols - deg, rows)
    col = (start[:, None] + np.arange(deg)[None, :]).astype(np.uint32).reshape(-1)
    val = (100 + rng.integers(-8, 9, rows * deg)).astype(np.float32)
    val[0] = 127
    Q = (100 + rng.integers(-8, 9, (nq, cols))).astype(np.float32)
    Q[:, 0] = 127
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=2048, k_max=k, max_batch=nq,
                 flags=E.FLAG_PROFILE, sample_stride=4)
    ns, cand = [], []
    for _ in range(4):
        eng.Q_reset(Q)
        eng.stats(reset=True)
        t = eng(k=k)
        assert eng.last_pass() == E.PASS_FILTER
        st = eng.stats(reset=True)
        ns.append(t)
        cand.append(st["cand_ms"] * 1e6)
    assert min(cand) > 0.5 * min(ns)


def test_exact_pass_of_more_queries_than_sms():
    rows, cols, nq, k = 20_000, 128, 333, 10
    ptr, col, val = E.gen_matrix(E.GEN_UNIFORM_DEG, rows, cols, 4, 10, seed=6)
    val = val - np.float32(0.4)
    Q = (np.random.default_rng(3).random((nq, cols)) * 2 - 1).astype(np.float32)
    eng = E.SpMV(rows, cols, ptr=ptr, col=col, val=val, bits=8, split=1, ck=64, k_max=k, max_batch=nq)
    eng.Q_reset(Q)
    idx, sc, _ = eng.run_exact(k=k)
    allrows = np.arange(rows, dtype=np.uint32)
    for i in range(0, nq, 37):
        ri, rs = orc.sort_tuples_f32(allrows, orc.rescore_f32(ptr, col, val, Q[i], allrows))
        assert np.array_equal(idx[i], ri[:k]) and np.array_equal(sc[i], rs[:k]), i
