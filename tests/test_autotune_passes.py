"""CPU tests of the tuner's choice among the passes, with a stand-in engine that tells which pass a run
took: the four-query pass is timed where it is the handle's own choice, and the filter only once."""
import time
import types

import numpy as np
import pytest

from acceles_gb300 import autotune as AT
from acceles_gb300 import engine as E


class FakeEngine:
    """Takes the pass that the engine would; a run sleeps per pass."""

    def __init__(self, nq, four_max, filtered):
        self.params = types.SimpleNamespace(flags=0, ck=256, split=1, batch_tile=0, sample_stride=0,
                                            max_batch=nq, k_max=5, batch_warps=0)
        self.four_max, self.filtered = four_max, filtered
        self.exact = np.arange(nq * 5, dtype=np.uint32).reshape(nq, 5)

    def retune(self, **kw):
        for key, v in kw.items():
            setattr(self.params, key, v)

    def info(self):
        return {"tensor_tiles": 0, "batch_warps": self.params.batch_warps or 16}

    def Q_reset(self, q):
        self.nq = len(q)

    def run_exact(self, k):
        return self.exact[: self.nq], None, 0

    def last_pass(self):
        tile = self.params.batch_tile
        if tile == 1:
            return E.PASS_PLAIN
        if tile == 0 and 1 < self.nq <= self.four_max:
            return E.PASS_FOUR
        return E.PASS_FILTER if self.filtered else E.PASS_DP4A

    def __call__(self, k):
        time.sleep({E.PASS_PLAIN: 0.008, E.PASS_FOUR: 0.001, E.PASS_DP4A: 0.004, E.PASS_FILTER: 0.002}[self.last_pass()])
        return 0

    def read_topk(self):
        return self.exact[: self.nq].copy(), None

    def stats(self, reset=False):
        return {"repaired": 0}


@pytest.mark.parametrize("nq,four_max,filtered,want,best", [
    (8, 48, False, {(1, 0), (0, 0)}, 0),                              # small batches: four queries per read
    (40, 48, False, {(1, 0), (0, 0), (128, 0), (128, 12), (128, 8)}, 0),
    (80, 48, False, {(1, 0), (128, 0), (128, 12), (128, 8)}, 128),    # (batch_tile 0 would be the dp4a pass)
    (80, 32, True, {(1, 0), (128, 0)}, 128),                          # the filter, once
])
def test_passes_timed(nq, four_max, filtered, want, best):
    eng = FakeEngine(nq, four_max, filtered)
    res = AT.tune(eng, np.zeros((nq, 8), np.float32), 5, ck_ladder=(256,), strides=(0,), reps=1)
    assert {(t["batch_tile"], t["batch_warps"]) for t in res["time_trials"]} == want
    assert res["params"]["batch_tile"] == best and eng.params.batch_tile == best
