"""Autotuner of the two-stage path for one resident matrix and one query workload, and the
batched sparse-query workload it was written for.

`tune()` works in two stages, both measured on the device through the handle's own calls:

1. Candidate count CK (per split): the smallest CK of a ladder whose two-stage Top-K equals
   the FP32-only single-stage Top-K (aes_run_exact: the same FP32 scores, the same
   (score desc, row desc) order) on at least `target` of the sample queries.  The rescoring
   is exact, so a query whose recall@K is 1 has an identical Top-K, and with split 1 a larger
   CK only adds candidates: the first CK that reaches the target is the smallest.
2. Sample stride and candidate pass: for each split's CK, every (stride, pass) of the grid is
   timed on the sample batch (wall time of aes_run, repairs included); the fastest wins.  The
   passes are the plain one (one query per matrix read), blocks of 128 queries, and the four-query
   pass where the handle's own choice (batch_tile 0) is that one.  Blocks are the dp4a pass, with 16
   (the most that fit at 1024 columns), 12 or 8 warps per CTA, or, where the handle holds the
   filter's layout and the sample is large enough, the filter, timed once (warps do not change
   it); for 4-bit matrices created with AES_FLAG_TENSOR also the tensor-core pass (FP8 tcgen05
   products of 128-row tiles; same results).  A handle holds the filter only for more than 64
   queries, so a sample of 64 or fewer chooses for batches of that size.

Every trial re-plans the handle with aes_retune; the packed matrix stays resident.

The reference has no tuner: its CK, split and bit width are compile-time constants of the
bitstream (types.hpp:39,148-149), and the method's accuracy scripts search the ReSparse ratio
for a fixed CK (search_best_resparse_ratio.py:55-117).

  python -m acceles_gb300.autotune [--rows 20000000] [--queries 256] [--tune-queries 32]

runs the batched sparse-query workload: a 20,000,000 x 1024 matrix with row degree
min(512, max(1, round(Gamma(shape 2, mean 32)))), uniform distinct columns, FP32 values
U(0,1), 4-bit per-row unsigned Ultra-CSR; 256 queries per step, each with its own density
drawn from U[5%, 30%] and values U(0,1); K = 100.
"""
from __future__ import annotations

import argparse
import json
import os
import time

import numpy as np

from . import engine as E

CK_LADDER = (128, 256, 512, 1024, 2048, 4096)
NO_ROW = 0xFFFFFFFF


def _recall(idx, exact, k):
    """Per-query |two-stage Top-K ∩ exact Top-K| / |exact Top-K|."""
    out = np.zeros(idx.shape[0])
    for i in range(idx.shape[0]):
        e = set(int(x) for x in exact[i, :k] if x != NO_ROW)
        g = set(int(x) for x in idx[i, :k] if x != NO_ROW)
        out[i] = len(e & g) / max(len(e), 1)
    return out


def _pass_of(eng, queries, k):
    """The form of the candidate pass that a run of `queries` takes; None where the engine cannot tell."""
    if not hasattr(eng, "last_pass"):
        return None
    eng.Q_reset(queries)
    eng(k=k)
    return eng.last_pass()


def _time_runs(eng, queries, k, reps):
    eng.Q_reset(queries)
    eng(k=k)  # warm: graphs, caches
    eng.stats(reset=True)
    best = float("inf")
    for _ in range(reps):
        t0 = time.perf_counter()
        eng(k=k)
        best = min(best, time.perf_counter() - t0)
    st = eng.stats(reset=True)
    return best, st["repaired"]


# (batch_tile, tensor cores, warps per CTA of the dp4a batched pass; 0 = the most that fit); batch_tile
# 0 stands for the four-query pass
PASSES = ((1, False, 0), (128, False, 0), (128, False, 12), (128, False, 8), (128, True, 0), (0, False, 0))


def tune(eng: E.SpMV, queries, k, ck_ladder=CK_LADDER, splits=(1,), strides=(0, 16, 64, 256),
         passes=PASSES, target=1.0, reps=3, log=None):
    """Choose CK, split, sample stride and candidate pass for `queries` (FP32 [nq, cols]) at
    K=k.  The returned params hold batch_tile, batch_warps and flags (AES_FLAG_TENSOR or 0).
    A pass is (batch_tile, tensor) or (batch_tile, tensor, batch_warps).

    Returns {"params": chosen aes_params fields, "ck_trials": [...], "time_trials": [...],
    "exact": the FP32-only Top-K rows of the sample}.  The handle is left retuned to the
    chosen parameters with max_batch = the sample's size.
    """
    Q = np.ascontiguousarray(np.atleast_2d(queries), np.float32)
    nq = Q.shape[0]
    base = eng.params.flags & ~E.FLAG_TENSOR
    eng.retune(max_batch=nq, k_max=max(k, 1), flags=base, batch_warps=0)
    eng.Q_reset(Q)
    exact, _, _ = eng.run_exact(k=k)

    ck_trials, chosen_ck = [], {}
    for split in splits:
        for ck in ck_ladder:
            if ck < split or (ck // split) * split > 4096:
                continue
            eng.retune(ck=ck, split=split, max_batch=nq, batch_tile=0, sample_stride=0)
            eng.Q_reset(Q)
            eng(k=k)
            idx, _ = eng.read_topk()
            rec = _recall(idx, exact, k)
            row = {"split": split, "ck": ck, "mean_recall": float(rec.mean()),
                   "frac_identical": float(np.mean(rec == 1.0))}
            ck_trials.append(row)
            if log:
                log(row)
            if row["frac_identical"] >= target:
                chosen_ck[split] = ck
                break
    if not chosen_ck:
        raise RuntimeError("no CK of the ladder reaches the recall target")

    time_trials = []
    best = None
    for split, ck in chosen_ck.items():
        for pas in passes:
            tile, tensor, warps = (tuple(pas) + (0,))[:3]
            if tile == 128 and nq < 16:
                continue
            flags = base | (E.FLAG_TENSOR if tensor else 0)
            for stride in strides:
                eng.retune(ck=ck, split=split, max_batch=nq, batch_tile=tile,
                           sample_stride=stride, flags=flags, batch_warps=warps)
                if tensor and not eng.info()["tensor_tiles"]:
                    break  # no tensor-core layout for this matrix or split
                if warps and eng.info()["batch_warps"] != warps:
                    break  # fewer warps fit: the trial of the most that fit covers it
                form = _pass_of(eng, Q, k) if (warps or tile == 0) else None
                if tile == 0 and form != E.PASS_FOUR:
                    break  # the handle's choice is one of the other passes
                if warps and form == E.PASS_FILTER:
                    break  # the filter, whatever the dp4a pass's warps
                sec, repaired = _time_runs(eng, Q, k, reps)
                row = {"split": split, "ck": ck, "batch_tile": tile, "tensor": tensor,
                       "batch_warps": warps, "sample_stride": stride,
                       "ms_per_query": sec * 1e3 / nq, "repaired": int(repaired)}
                time_trials.append(row)
                if log:
                    log(row)
                if best is None or row["ms_per_query"] < best["ms_per_query"]:
                    best = row
    params = {"ck": best["ck"], "split": best["split"], "batch_tile": best["batch_tile"],
              "sample_stride": best["sample_stride"], "batch_warps": best["batch_warps"],
              "flags": base | (E.FLAG_TENSOR if best["tensor"] else 0)}
    eng.retune(max_batch=nq, **params)
    return {"params": params, "ck_trials": ck_trials, "time_trials": time_trials,
            "exact": exact}


def sparse_queries(n, cols, seed, lo=0.05, hi=0.30):
    """n FP32 queries, query i with density d_i ~ U[lo, hi] and values U(0,1)."""
    rng = np.random.default_rng(seed)
    Q = rng.random((n, cols)).astype(np.float32)
    d = rng.uniform(lo, hi, n)
    Q[rng.random((n, cols)) >= d[:, None]] = 0.0
    return Q


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--rows", type=int, default=20_000_000)
    ap.add_argument("--cols", type=int, default=1024)
    ap.add_argument("--queries", type=int, default=256)
    ap.add_argument("--tune-queries", type=int, default=64)
    ap.add_argument("--k", type=int, default=100)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--seed", type=int, default=4242)
    ap.add_argument("--json", default=None, help="also write the result lines here")
    args = ap.parse_args()
    peak = 6800.0
    pk = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "MEASURED_PEAKS.json")
    bf16 = 1900.0  # TFLOP/s, fallback; FP8 dense is taken as twice the measured bf16 rate
    if os.path.exists(pk):
        mp = json.load(open(pk))
        peak = float(mp["hbm_gbs"])
        bf16 = float(mp.get("bf16_tflops", bf16))
    lines = []

    def emit(d):
        lines.append(d)
        print(json.dumps(d), flush=True)

    t0 = time.perf_counter()
    ptr, col, val = E.gen_matrix(E.GEN_GAMMA_DEG, args.rows, args.cols, 32, 512, seed=args.seed)
    t_gen = time.perf_counter() - t0
    t0 = time.perf_counter()
    eng = E.SpMV(args.rows, args.cols, ptr=ptr, col=col, val=val, bits=4,
                 quant=E.QUANT_UNSIGNED_ROW, split=1, ck=1024, k_max=args.k,
                 max_batch=args.queries, flags=E.FLAG_GRAPHS | E.FLAG_TENSOR)
    t_build = time.perf_counter() - t0
    info = eng.info()
    emit({"matrix": f"{args.rows}x{args.cols} gamma(2, mean 32) cap 512, U(0,1), 4-bit per-row "
                    "unsigned", "nnz": info["nnz"], "packets": info["packets"],
          "packet_bytes": info["packet_bytes"], "device_bytes": info["device_bytes"],
          "gen_s": t_gen, "build_s": t_build})

    tuneQ = sparse_queries(args.tune_queries, args.cols, args.seed + 1)
    res = tune(eng, tuneQ, args.k, log=lambda r: emit({"trial": r}))
    prm = res["params"]
    emit({"chosen": prm})

    # measure the chosen configuration on the workload's own queries
    Q = sparse_queries(args.queries * 2, args.cols, args.seed + 2)
    nq = args.queries
    tflag = prm["flags"] & E.FLAG_TENSOR
    run_prm = {k: v for k, v in prm.items() if k != "flags"}
    eng.retune(max_batch=nq, flags=E.FLAG_GRAPHS | tflag, **run_prm)
    for s in range(args.warmup):
        eng.Q_reset(Q[(s % 2) * nq:(s % 2 + 1) * nq])
        eng(k=args.k)
    dev_ns, wall = 0, 0.0
    for s in range(args.steps):
        eng.Q_reset(Q[(s % 2) * nq:(s % 2 + 1) * nq])
        t0 = time.perf_counter()
        dev_ns += eng(k=args.k)
        wall += time.perf_counter() - t0
    st = eng.stats(reset=True)
    qps_dev = args.steps * nq / (dev_ns / 1e9)
    qps_e2e = args.steps * nq / wall
    # candidate-pass launch time, profiled outside graphs
    eng.retune(max_batch=nq, flags=E.FLAG_PROFILE | tflag, **run_prm)
    eng.Q_reset(Q[:nq])
    eng(k=args.k)
    eng.stats(reset=True)
    eng(k=args.k)
    stp = eng.stats(reset=True)
    launches = max(stp["cand_timed"], 1)
    launch_ms = stp["cand_ms"] / launches
    q_launch = nq / launches  # queries one launch scores (tensor cores: 256 on CTA pairs)
    kpad = (args.cols + 31) // 32 * 32
    rtiles = (args.rows + 127) // 128
    if tflag:
        # tensor-core pass: 4-byte entries, chunk offsets, the e4m3 query operands; dense FP8
        # products of every 128-row tile with the launch's queries
        alg = info["quantized_nnz"] * 4 + (rtiles * ((kpad + 255) // 256) + 1) * 4 + q_launch * kpad
        flops = 2.0 * rtiles * 128 * q_launch * kpad
    else:
        alg = info["packets"] * 64 + (info["tiles"] + 1) * 4 + args.cols * {128: 128, 0: 4}.get(prm["batch_tile"], 1)
        flops = None
    gbs = alg / (launch_ms / 1e3) / 1e9
    # recall of the measured queries against the FP32-only Top-K
    idx, _ = eng.read_topk()
    eng.retune(max_batch=nq, flags=0, **run_prm)
    eng.Q_reset(Q[:nq])
    exact, _, _ = eng.run_exact(k=args.k)
    rec = _recall(idx, exact, args.k)
    emit({"workload": "batched sparse queries, 20Mx1024 gamma deg, 4-bit", "queries_per_step": nq,
          "steps": args.steps, "qps_device": qps_dev, "qps_e2e_host_buffers": qps_e2e,
          "ms_per_step_device": dev_ns / 1e6 / args.steps, "repaired": st["repaired"],
          "cand_pass": {"launch_ms": launch_ms, "queries_per_launch": q_launch,
                        "ms_per_128_queries": launch_ms * 128 / q_launch, "alg_bytes": alg, "gbs": gbs,
                        "frac_of_measured_hbm": gbs / peak, "tensor_cores": bool(tflag),
                        "dense_tflops": (flops / (launch_ms / 1e3) / 1e12) if flops else None,
                        "frac_of_fp8_dense": ((flops / (launch_ms / 1e3) / 1e12) / (2 * bf16))
                        if flops else None},
          "recall_at_k_mean": float(rec.mean()), "frac_identical_to_fp32_exact": float(np.mean(rec == 1.0)),
          "params": prm})
    if args.json:
        with open(args.json, "w") as f:
            for l in lines:
                f.write(json.dumps(l) + "\n")
    eng.close()


if __name__ == "__main__":
    main()
