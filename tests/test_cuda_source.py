"""CPU checks of the CUDA sources for rules that no run shows: kernels launched while their predecessor
still runs read what it writes through coherent loads only."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "acceles_gb300", "csrc")


def _src(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


# arrays of the matrix and of the handle's configuration: nothing writes them while a batch runs
RESIDENT = {"a.rowscale", "a.rowstat", "a.tile_rowbase", "a.sample_first", "a.ptr", "a.val", "a.col", "ent",
            "part_begin", "r_part", "a.csr_ptr", "a.csr_col", "a.csr_val", "src[w]", "src"}
PLAIN_LAUNCH = {"k_recheck": {"a.thr"}}  # waits for its predecessor's end


def _kernels(text):
    """name -> (parameter list, body up to the next kernel)"""
    heads = list(re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", text))
    out = {}
    for h, nxt in zip(heads, heads[1:] + [None]):
        end = nxt.start() if nxt else len(text)
        out[h.group(1)] = (text[h.end():text.index(")", h.end())], text[h.end():end])
    return out


def _chained():
    eng = _src("aes_engine.cu")
    names = set(re.findall(r"chain\(\s*(k_\w+)", eng)) | {"k_threshold_warp"}
    if re.search(r"chain\(\s*(?:aes::)?pick_plain", eng):
        names.add("k_cand_plain")
    if re.search(r"chain\(\s*pick_batch", eng):
        names.add("k_cand_batch")
    return names | {"k_cand_multi", "k_cand_tc"}


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cuh")))
def test_read_only_loads_are_of_resident_arrays(name):
    text = _src(name)
    plain = {a for k, s in PLAIN_LAUNCH.items() if k + "(" in text for a in s}
    for m in re.finditer(r"__ldg\(\s*([\w.]+(?:\[w\])?)", text):
        assert m.group(1) in RESIDENT | plain, (name, m.group(0), text.count("\n", 0, m.start()) + 1)


def test_dependent_kernels_take_no_read_only_parameters():
    kernels = {}
    for f in os.listdir(CSRC):
        if f.endswith(".cuh"):
            kernels.update(_kernels(_src(f)))
    chained = _chained()
    assert {"k_threshold", "k_select", "k_final", "k_qtable", "k_tf_qstats", "k_keys_transpose"} <= chained
    for k in chained:
        for p in re.findall(r"const\s+\w+\*\s+__restrict__\s+(\w+)", kernels[k][0]):
            assert p in RESIDENT, (k, p)
        assert "grid_wait();" in kernels[k][1], k


def test_pair_barriers_are_used_at_cluster_scope():
    """What crosses the CTAs of a pair is handed over at cluster scope; a barrier operation without a
    scope orders the threads of one CTA only."""
    text = _src("aes_tc.cuh")
    arrives = re.findall(r"mbarrier\.arrive([.\w:]*)\.b64", text)
    assert any("shared::cluster" in a for a in arrives)
    for a in arrives:
        if "shared::cluster" in a:
            assert re.match(r"\.(release|relaxed)\.cluster\.", a), a
    # relaxed ones stand behind a fence: of shared memory where bytes are handed over, else tcgen05's
    hand = text[text.index("void tc_arrive_warp"):]
    hand = hand[:hand.index("\n}\n")]
    assert "if constexpr (BYTES) asm volatile(\"fence.release.sync_restrict::shared::cta.cluster;\"" in hand
    assert hand.index("fence.release") < hand.index("mbarrier.arrive.relaxed.cluster")
    assert re.search(r"tc_fence_before\(\);\s+tc_arrive_warp<PAIR, false>\(empty\)", text)
    assert "tc_arrive_warp<true, true>(b_staged" in text
    assert "if (done) asm volatile(\"fence.acquire.sync_restrict::shared::cluster.cluster;\"" in text
    body = text[text.index("k_cand_tc(TcArgs a)"):]
    waits = re.findall(r"tc_wait(?:_own)?(<\w+>)?\((b_\w+)", body)
    for scope, bar in waits:
        if bar in ("b_done", "b_full", "b_empty"):
            assert scope in ("<kAcq>", "<kRlx>"), (bar, scope)
    staged = [scope for scope, bar in waits if bar == "b_staged"]
    assert sorted(staged) == ["", "<kAcq>"], staged  # the odd CTA's own phases; the MMA role's


def test_k_final_is_dependent_only_where_one_wave_holds_it():
    """A dependent kernel of several large CTAs per SM may get one (Engine::chain): k_final is launched
    so in one place, which looks at its size."""
    eng = _src("aes_engine.cu")
    at = [m.start() for m in re.finditer(r"chain\(k_final", eng)]
    assert len(at) == 1
    assert "<= (uint32_t)sm_count) {" in eng[at[0] - 80:at[0]]
