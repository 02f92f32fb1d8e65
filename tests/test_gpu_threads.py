"""Calls from several Python threads."""
import threading

import pytest

from tests import gpu_utils as G
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _call(ops, mu, L, M):
    """A call of the operator (through the dispatcher, which lets go of the interpreter lock) and its arguments' owner."""
    import torch
    from vllm_b200 import _custom_ops
    a = G.t16(H.make_activations(M, L.size_k, L.dtype), L.dtype)
    op = getattr(torch.ops, _custom_ops.ops_namespace()).gptq_marlin_gemm
    args = (a, None, G.ti32(L.marlin_q), None, G.t16(L.marlin_s, L.dtype), None, G.ti32(L.marlin_zp), G.ti32(L.g_idx),
            G.ti32(L.sort_idx), mu.marlin_make_workspace_new(torch.device("cuda")), L.type_id, M, L.size_n, L.size_k,
            True, False, True, False)
    return lambda: op(*args)


def test_threads_share_a_stream():
    """Act-order calls of several threads on one stream: each gathers its rows into the stream's scratch and multiplies
    them from there, with partial sums of different sizes behind."""
    import torch
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import marlin_utils as mu
    calls = [_call(ops, mu, H.make_layer(K, N, "uint4b8", 128, True, "float16"), M)
             for M, K, N in ((3, 1024, 512), (40, 2048, 1024), (200, 1024, 2048), (64, 4096, 512))]
    want = [c() for c in calls]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        outs = [calls[i]() for _ in range(100)]
        wrong.extend(i for o in outs if not torch.equal(o, want[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_direct_call_lets_other_threads_run():
    """While the direct call allocates and launches (and waits for room in the launch queue) another Python thread
    gets the interpreter.  With a switch interval of minutes it does so only when the call gives it up."""
    import sys
    import time

    import torch
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import marlin_utils as mu
    M, K, N = 4096, 8192, 128
    gen = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randint(-2**31, 2**31 - 1, (K // 16, N * 2), dtype=torch.int32, device="cuda", generator=gen)
    s = (torch.rand((K // 128, N), device="cuda", generator=gen) * 0.018 + 0.002).half()
    a = torch.randn((M, K), device="cuda", dtype=torch.float16, generator=gen)
    e = torch.empty(0, dtype=torch.int32, device="cuda")
    args = (a, q, None, s, None, e, e, e, mu.marlin_make_workspace_new(torch.device("cuda")), mu.scalar_types.uint4b8.id,
            -1, N, K, ops.K_FULL)
    assert ops._linear(*args) is not None
    turns, stop = [0], threading.Event()

    def other():
        while not stop.is_set():
            turns[0] += 1
            time.sleep(0)       # gives the interpreter back

    interval = sys.getswitchinterval()
    thread = threading.Thread(target=other)
    try:
        sys.setswitchinterval(600)
        thread.start()
        outs = [None] * 3000    # more calls than the launch queue holds; kept, since freeing a tensor may switch threads
        before = turns[0]
        for i in range(len(outs)):
            outs[i] = ops._linear(*args)
        during = turns[0] - before
    finally:
        sys.setswitchinterval(interval)
        stop.set()
        thread.join()
    torch.cuda.synchronize()
    assert during > 0
