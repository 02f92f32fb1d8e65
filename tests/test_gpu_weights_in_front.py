"""A layer's weights written by the kernels directly in front of a call, with nothing between: weights and scales replaced by
ordinary copies at every row count, and above 128 rows scales that come from a kernel which lets the next one start early
(RMSNorm's output).  The results are those of the new values, call after call."""
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu
K, N, GROUP = 1024, 4096, 128


def _setup(M, dtype="bfloat16"):
    import torch
    from tests import gpu_utils as G
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import marlin_utils as mu
    from vllm_b200.scalar_type import ScalarType
    layers = [H.make_layer(K, N, "uint4b8", GROUP, False, dtype, seed=s) for s in range(3)]
    qs = [G.ti32(L.marlin_q) for L in layers]
    ss = [G.t16(L.marlin_s, dtype) for L in layers]
    x = G.t16(H.make_activations(M, K, dtype), dtype)
    q, s = torch.empty_like(qs[0]), torch.empty_like(ss[0])
    ws = mu.marlin_make_workspace_new(torch.device("cuda"))
    none = torch.empty(0, dtype=torch.int32, device="cuda")

    def gemm(q, s):
        return ops.gptq_marlin_gemm(x, None, q, None, s, None, none, none, none, ws, ScalarType.from_id(layers[0].type_id), M, N, K,
                                    is_k_full=True, use_fp32_reduce=True, is_zp_float=False)

    return torch, ops, qs, ss, q, s, gemm


@pytest.mark.parametrize("M", [1, 24, 64, 128, 129, 300])
def test_copies_in_front(M):
    torch, ops, qs, ss, q, s, gemm = _setup(M)
    want = [gemm(a, b) for a, b in zip(qs, ss)]
    torch.cuda.synchronize()
    got = []
    for i in range(12):
        q.copy_(qs[i % 3])
        s.copy_(ss[i % 3])
        got.append(gemm(q, s))
    torch.cuda.synchronize()
    assert all(bool(torch.equal(g, want[i % 3])) for i, g in enumerate(got))


@pytest.mark.parametrize("M", [129, 160, 300, 700])
def test_writer_that_lets_the_call_start_early(M):
    torch, ops, qs, ss, q, s, gemm = _setup(M)
    gain = torch.full((N,), 0.01, dtype=s.dtype, device="cuda")
    raw = [torch.randn(K // GROUP, N, device="cuda").to(s.dtype) for _ in range(3)]
    scales = []
    for r in raw:
        t = torch.empty_like(s)
        ops.rms_norm(t, r, gain, 1e-5)
        scales.append(t)
    torch.cuda.synchronize()
    want = [gemm(qs[0], t) for t in scales]
    torch.cuda.synchronize()
    got = []
    for i in range(12):
        ops.rms_norm(s, raw[i % 3], gain, 1e-5)
        got.append(gemm(qs[0], s))
    torch.cuda.synchronize()
    assert all(bool(torch.equal(g, want[i % 3])) for i, g in enumerate(got))
