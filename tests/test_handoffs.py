"""Order of the hand-offs in the tensor-core kernel, read from its source: a missing fence shows in no result, or in one
of many thousand, so that running the kernel is no test of it."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vllm_b200", "csrc", "gemm_tc.cuh")


def _code():
    with open(SRC) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_weight_slots_go_back_behind_a_proxy_fence():
    """The producer refills a weight slot with a copy (async proxy): between the last read of a slot and the arrival
    that gives it back stand the proxy fence of every reading lane and, after it, the warp barrier."""
    code = _code()
    dequant = code[code.index("mbar_wait<false>(full_w"):]
    arrivals = [m.start() for m in re.finditer(r"mbar_arrive\(empty_w\(", dequant)]
    assert arrivals and "mbar_arrive(empty_w(" not in code[:code.index("mbar_wait<false>(full_w")]
    for at in arrivals:
        before = dequant[:at]
        read = max(before.rfind("lds128("), before.rfind("lds32("))
        fence, sync = before.rfind("fence_proxy_async_smem();"), before.rfind("__syncwarp();")
        assert read < fence < sync


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
    wait = re.search(r'if \(!p\.weights_ahead\) asm volatile\("griddepcontrol\.wait;', producer)
    assert wait and wait.start() < producer.index("tma_load")
    with open(os.path.join(os.path.dirname(SRC), "gemm_tc.cu")) as f:
        assert re.findall(r"weights_ahead = ([^;]*);", f.read()) == ["size_m <= 128"]
