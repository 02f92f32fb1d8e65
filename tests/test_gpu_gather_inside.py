"""Act-order at up to eight rows: the decode kernel gathers its part of A itself where that is at most eight k of one row
for each of its 256 threads.  Both sides of that line, ragged splits of K, every row count, a strided A and a permutation
that is not aligned (which takes the gather kernel); the two ways give the same bits."""
import pytest

from oracle import marlin_oracle as mo
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N,qtype,group,dtype", [
    (1, 128, 64, "uint4b8", 32, "bfloat16"),         # one CTA a slice
    (1, 1040, 192, "uint4b8", 16, "float16"),        # 65 k-tiles: parts of eight and nine
    (3, 1152, 128, "uint4b8", 64, "bfloat16"),
    (5, 2048, 320, "uint8b128", 128, "float16"),
    (7, 2048, 256, "uint4b8", 128, "float16"),
    (8, 2048, 256, "uint4b8", 128, "bfloat16"),      # the last that fits: 32 pieces of eight rows
    (8, 2176, 256, "uint4b8", 64, "bfloat16"),       # beyond
    (2, 8192, 256, "uint8b128", 128, "bfloat16"),
    (1, 14336, 128, "uint4b8", 128, "bfloat16"),
])
def test_gather_inside(M, K, N, qtype, group, dtype):
    import torch
    from tests import gpu_utils as G
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import marlin_utils as mu
    from vllm_b200.scalar_type import ScalarType
    L = H.make_layer(K, N, qtype, group, True, dtype, with_bias=M % 2 == 1)
    a = H.make_activations(M, K, dtype)
    out = G.run_gemm(ops, mu, L, a)
    max_frac, mean_rel = H.gemm_errors(out, mo.gemm_ref(a, L.w, L.bias))
    assert max_frac <= H.MAX_ABS_FRAC and mean_rel <= H.MEAN_REL, (max_frac, mean_rel)
    ws = mu.marlin_make_workspace_new(torch.device("cuda"))
    bias = None if L.marlin_bias is None else G.t16(L.marlin_bias, dtype)
    perm, q, s = G.ti32(L.sort_idx), G.ti32(L.marlin_q), G.t16(L.marlin_s, dtype)

    def gemm(x, g_idx, order):
        y = ops.gptq_marlin_gemm(x, None, q, bias, s, None, None, g_idx, order, ws, ScalarType.from_id(L.type_id), M, N, K,
                                 is_k_full=True, use_fp32_reduce=True, is_zp_float=False)
        return G.n16(y)

    x = G.t16(a, dtype)
    none = torch.empty(0, dtype=torch.int32, device="cuda")
    front = gemm(x[:, perm.long()].contiguous(), none, none)   # the columns gathered in front
    assert (front == out).all()
    wide = torch.zeros((M, K + 24), dtype=x.dtype, device="cuda")
    wide[:, 8:K + 8] = x
    assert (gemm(wide[:, 8:K + 8], G.ti32(L.g_idx), perm) == out).all()
    odd = torch.empty(K + 1, dtype=torch.int32, device="cuda")[1:].copy_(perm)
    assert (gemm(x, G.ti32(L.g_idx), odd) == out).all()
