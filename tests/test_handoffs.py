"""Order of the hand-offs in the tensor-core kernel, read from its source: a missing fence shows in no result, or in one
of many thousand, so that running the kernel is no test of it."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vllm_b200", "csrc", "gemm_tc.cuh")


def _code():
    with open(SRC) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _body(code, head):
    """What stands between the braces that `head` opens."""
    at = code.index(head) + len(head)
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(code[end], 0)
        end += 1
    return code[at:end - 1]


def _in_order(text, *steps):
    """Every step is there, and all of one stand in front of all of the next."""
    found = [[m.start() for m in re.finditer(s, text)] for s in steps]
    assert all(found), [s for s, f in zip(steps, found) if not f]
    for (s0, f0), (s1, f1) in zip(zip(steps, found), list(zip(steps, found))[1:]):
        assert f0[-1] < f1[0], (s0, s1)


def _dequant(code):
    """The dequant warps' part and its three ways of keeping converted weights: rounds held in registers, TMEM, shared
    memory."""
    part = _body(code, "} else if (warp < kDequantWarps) {")
    hold = _body(part, "if constexpr (Cfg::kHoldRound) {\n          uint32_t f0")
    in_tmem = "} else if constexpr (Cfg::kInTmem) {"
    in_smem = part[part.index(in_tmem) + len(in_tmem) + len(_body(part, in_tmem)):]
    assert in_smem.startswith("} else {")
    return part, hold, _body(part, in_tmem), _body(in_smem, "} else {")


def check_weight_slots(code):
    """The producer refills a weight slot with a copy (async proxy): between the last read of a slot and the arrival
    that gives it back stand the proxy fence of every reading lane and, after it, the warp barrier."""
    part, hold, tmem, smem = _dequant(code)
    assert len(re.findall(r"mbar_arrive\w*\(empty_w", code)) == 1
    _in_order(_body(part, "auto give_back = [&]() {"), r"fence_proxy_async_smem\(\);", r"__syncwarp\(\);", r"mbar_arrive\(empty_w\(")
    # the reads: in shared memory's own way plain, in the others inside convert(), of both steps of the round
    step = _body(part, "auto convert_step = [&](int st, uint32_t (&f)[32], auto scaled_c) {")
    reads = r"\blds\d+\("
    assert len(re.findall(reads, part)) == len(re.findall(reads, step + smem))
    _in_order(hold, r"\bconvert\(", r"give_back\(\);")
    _in_order(tmem, r"\bconvert\(st", r"if \(st == 1\) \{\s*give_back\(\);")
    _in_order(smem, r"\blds\d+\(", r"give_back\(\);")
    assert [len(re.findall(r"give_back\(\)", t)) for t in (part, hold, tmem, smem)] == [3, 1, 1, 1]


def check_converted_weights(code):
    """Converted weights are written once the MMAs that read their place have retired, are complete before the fence, and
    the fence stands before the arrival that the MMA warp waits for."""
    part, hold, tmem, smem = _dequant(code)
    for way in (hold, tmem):
        _in_order(way, r"wait_empty\(\)", r"tc_fence_after\(\);", r"tmem_st32\(", r"tmem_st_wait\(\);", r"tc_fence_before\(\);")
    _in_order(smem, r"wait_empty\(\)", r"stmatrix_x4_off", r"fence_proxy_async_smem\(\);")
    rest = part[part.index(smem) + len(smem):]
    _in_order(rest, r"__syncwarp\(\);", r"mbar_arrive\(full\(ring\.i\)")
    assert len(re.findall(r"mbar_arrive\w*\(full\(", code)) == 1
    mma = _body(code, "} else if (warp == kMmaWarp) {")
    leader, relay = _body(mma, "if (rank == 0) {"), mma[mma.index("const uint32_t leader"):]
    loop = _body(leader, "for (int r = sg.r0; r < sg.r1; ++r) {")
    _in_order(loop, r"mbar_wait<kPair>\(full\(", r"tc_fence_after\(\);", r"\bissue\(")
    _in_order(relay, r"mbar_wait<false>\(full\(", r"tc_fence_after\(\);", r"tc_fence_before\(\);", r"mbar_arrive_cluster\(leader")


def check_accumulators(code):
    """The epilogue reads a buffer behind the wait and its fence, and gives it back when the values are in registers."""
    epi = code[code.index("auto take = [&]() {"):]
    _in_order(_body(epi, "auto take = [&]() {"), r"mbar_wait<kPair", r"tc_fence_after\(\);")
    _in_order(_body(epi, "auto release = [&]() {"), r"tc_fence_before\(\);", r"__syncwarp\(\);", r"mbar_arrive\w*\(")
    _in_order(_body(epi, "if constexpr (!SUMS) {"), r"take\(\);", r"tmem_ld32\(", r"tmem_ld_wait\(\);", r"release\(\);")
    _in_order(_body(epi, "for (int b = 0; b < NB; ++b) {"), r"tmem_ld_wait\(\);", r"release\(\);")


CHECKS = (check_weight_slots, check_converted_weights, check_accumulators)


@pytest.mark.parametrize("check", CHECKS, ids=lambda c: c.__name__)
def test_order(check):
    check(_code())


@pytest.mark.parametrize("check,old,new", [
    (check_weight_slots, "if (mine0) convert(0, f0);", "give_back(); if (mine0) convert(0, f0);"),
    (check_weight_slots, "if (mine1) convert(1, f1);\n          give_back();", "give_back();\n if (mine1) convert(1, f1);"),
    (check_weight_slots, "if (mine) convert(st, f);\n            if (st == 1) {\n              give_back();",
     "if (st == 1) give_back();\n if (mine) convert(st, f);\n if (st == 1) {"),
    (check_weight_slots, "if (st == 1) {\n              give_back();", "if (st == 0) {\n              give_back();"),
    (check_weight_slots, "uint32_t w2[2][NW]", "give_back(); uint32_t w2[2][NW]"),
    (check_weight_slots, "fence_proxy_async_smem();\n          __syncwarp();\n          mbar_arrive(empty_w",
     "__syncwarp();\n          mbar_arrive(empty_w"),
    (check_weight_slots, "__syncwarp();\n          mbar_arrive(empty_w", "mbar_arrive(empty_w"),
    (check_converted_weights, "tmem_st_wait();", ""),
    (check_converted_weights, "tmem_st_wait();\n          tc_fence_before();", "tc_fence_before();\n tmem_st_wait();"),
    (check_converted_weights, "tc_fence_before();\n        } else {", "} else {"),
    (check_converted_weights, "tc_fence_after();\n          if (mine0) tmem_st32", "if (mine0) tmem_st32"),
    (check_converted_weights, "fence_proxy_async_smem();  ", ""),
    (check_converted_weights, "tc_fence_after();\n              tc_fence_before();", ""),
    (check_converted_weights, "tc_fence_after();\n            const uint32_t da", "const uint32_t da"),
    (check_accumulators, "else release();", ";"),
    (check_accumulators, "tmem_ld_wait();\n              if (b + 1", "if (b + 1"),
])
def test_a_broken_order_is_seen(check, old, new):
    code = _code()
    assert old in code
    with pytest.raises(AssertionError):
        check(code.replace(old, new))


def test_arrivals_at_the_other_cta_release_at_cluster_scope():
    """What the second CTA of a pair has stored is read by the first one's MMA: the arrival that says so is a release
    at cluster scope, and the waits on the barriers that the pair shares acquire at cluster scope."""
    code = _code()
    remote = [m.start() for m in re.finditer(r"mbarrier\.arrive[\w.]*\.shared::cluster", code)]
    assert len(remote) == 1
    body = code[code.rfind("__device__", 0, remote[0]):remote[0] + 80]
    assert "mbar_arrive_cluster" in body
    assert body.index("fence.release.sync_restrict::shared::cta.cluster") < body.index("mbarrier.arrive.relaxed.cluster")
    assert "try_wait.parity.acquire.cluster" in code
    mma = code[code.index("warp == kMmaWarp) {"):code.index("warp < kDequantWarps) {")]
    assert "mbar_wait<kPair>(full(" in mma and "mbar_wait<kPair>(tmem_empty(" in mma


def test_weights_of_prompts_are_fetched_behind_the_wait():
    """What a kernel in front writes is visible after griddepcontrol.wait alone: above 128 rows, where calls make no
    exception for a layer's constants, the producer waits before its first copy."""
    code = _code()
    producer = code[code.index("warp == kProducerWarp) {"):code.index("warp == kTokenWarp) {")]
    wait = re.search(r'if \(p\.m > kAheadRows\) asm volatile\("griddepcontrol\.wait;', producer)
    assert wait and wait.start() < producer.index("tma_load") and "constexpr int kAheadRows = 128;" in code
