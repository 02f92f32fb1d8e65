"""The all-reduce in the decode GEMM's epilogue, on one GPU: what the other rank would have sent is in this rank's receive
buffer before the call, so that no kernel waits.  The output is the sum in rank order, rounded once, of the two ranks' rounded
parts, and the packets that this rank sends are the GEMM's output, every one, whichever CTA of a cluster owns a column: all
cluster sizes, columns (up to eight rows) and 8-row blocks shared out, act-order gathered inside and in front, both ranks,
three calls in a row (both parities of the buffer, a flag used again)."""
import types

import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
WORLD = 2


@pytest.mark.parametrize("rank", [0, 1])
@pytest.mark.parametrize("M,K,N,qtype,group,act,dtype", [
    (1, 2048, 256, "uint4b8", 128, True, "bfloat16"),     # gathered inside, clusters of eight
    (5, 1040, 192, "uint4b8", 16, True, "float16"),       # ragged parts, one-tile slices
    (8, 2048, 256, "uint4b8", 128, True, "bfloat16"),
    (8, 2176, 256, "uint4b8", 64, True, "float16"),       # gathered in front
    (1, 128, 64, "uint4b8", 32, True, "bfloat16"),        # one CTA a slice
    (7, 512, 4608, "uint4", 128, False, "float16"),       # clusters of two or four
    (3, 1024, 1024, "uint4b8", -1, False, "bfloat16"),
    (4, 256, 19456, "uint4b8", 64, False, "bfloat16"),    # more slices than SMs
    (12, 2048, 1024, "uint4b8", 32, True, "bfloat16"),    # 8-row blocks shared out
    (32, 1024, 256, "uint4b8", 32, False, "float16"),
    (16, 1024, 1024, "uint4b8", 128, False, "bfloat16"),  # the shard that the two-GPU test compares with GEMM + all-reduce
    (32, 1024, 1024, "uint4b8", 128, False, "bfloat16"),
])
def test_epilogue_sums_what_the_other_rank_sent(M, K, N, qtype, group, act, dtype, rank):
    import torch
    from tests import gpu_utils as G
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import _lib
    from vllm_b200 import marlin_utils as mu
    from vllm_b200.scalar_type import ScalarType
    lib = _lib.load()
    L = H.make_layer(K, N, qtype, group, act, dtype)
    x = G.t16(H.make_activations(M, K, dtype), dtype)
    ws = mu.marlin_make_workspace_new(x.device)
    args = (None, G.ti32(L.marlin_q), None, G.t16(L.marlin_s, dtype), None, G.ti32(L.marlin_zp), G.ti32(L.g_idx), G.ti32(L.sort_idx),
            ws, ScalarType.from_id(L.type_id), M, N, K)
    flags = dict(is_k_full=True, use_fp32_reduce=True, is_zp_float=False)
    most = M * N * 2
    bufs = [torch.zeros(lib.b200q_all_reduce_buffer_bytes(WORLD, most) // 4, dtype=torch.int32, device="cuda") for _ in range(WORLD)]
    slots = [b[:2 * WORLD * most // 2].view(2, WORLD, M * N // 2, 2) for b in bufs]   # [parity][sender][packet]{values, flag}
    link = types.SimpleNamespace(peer_ptrs=torch.tensor([b.data_ptr() for b in bufs], dtype=torch.int64, device="cuda"),
                                 state=torch.zeros(lib.b200q_all_reduce_state_bytes() // 4, dtype=torch.int32, device="cuda"),
                                 rank=rank, world_size=WORLD, max_size=most)
    peer = 1 - rank
    assert lib.b200q_device_error(1) == 0
    lib.b200q_all_reduce_set_poll_limit(2000)
    try:
        for call in range(3):
            a = torch.roll(x, call, 0) * (1 + call)
            mine = ops.gptq_marlin_gemm(a, *args, **flags)
            theirs = torch.randn(M, N, device="cuda").to(x.dtype) * mine.float().std().to(x.dtype)
            parity, flag = call & 1, (call >> 1) + 1
            slots[rank][parity, peer, :, 0] = theirs.view(torch.int32).flatten()
            slots[rank][parity, peer, :, 1] = flag
            out = ops.gptq_marlin_gemm(a, *args, **flags, reduce_link=link)
            torch.cuda.synchronize()
            assert lib.b200q_device_error(1) == 0
            assert torch.equal(out, (mine.float() + theirs.float()).to(x.dtype))
            sent = slots[peer][parity, rank]
            assert torch.equal(sent[:, 0], mine.view(torch.int32).flatten()) and bool((sent[:, 1] == flag).all())
            assert link.state[:2].tolist() == [call + 1, 0]
    finally:
        lib.b200q_all_reduce_set_poll_limit(0)
