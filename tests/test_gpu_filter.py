"""GPU tests of the tensor-core filter (6- and 8-bit batches) beside its forms: rows and values at
its edges, its memory, and how it gives way to the dp4a pass.  Results must equal the oracle's."""
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
