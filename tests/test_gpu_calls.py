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
