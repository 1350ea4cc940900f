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
