"""Group scales stay out of the 16-bit products wherever a call may take the decode kernel: up to 32 rows, and in
mixture-of-experts layers of any size.  Results are compared with 64-bit sums of the unrounded weights."""
import numpy as np
import pytest

from oracle import marlin_oracle as mo
from tests import gpu_utils as G
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _weights64(L):
    q = L.q.astype(np.float64) - (0 if L.has_zp else L.type_bias)
    reps = L.size_k // L.num_groups
    if L.has_zp:
        q = q - np.repeat(L.zeros, reps, axis=0)
    return q * np.repeat(L.scales.astype(np.float64), reps, axis=0)


@pytest.mark.parametrize("M,K,N,qtype,group,dtype", [
    (24, 4096, 1024, "uint4b8", 128, "bfloat16"),
    (32, 4096, 1024, "uint8b128", 128, "bfloat16"),
    (24, 5504, 2560, "uint4b8", 128, "float16"),
    (32, 3456, 9024, "uint8b128", 128, "float16"),    # half a column tile at the end
    (16, 7168, 9024, "uint8b128", 64, "float16"),     # two groups a round
    (32, 7168, 9024, "uint4b8", 1024, "bfloat16"),    # k-shares that begin inside a group
    (17, 11008, 5120, "uint4", 128, "float16"),
    (8, 11072, 5120, "uint8", 64, "bfloat16"),        # an odd number of steps
    (31, 4096, 9024, "uint4b8", 32, "bfloat16"),      # groups that the tensor-core kernel does not take
    (32, 8064, 5120, "uint8b128", 192, "float16"),
])
def test_few_rows_keep_group_scales_in_fp32(M, K, N, qtype, group, dtype):
    import torch
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import _lib
    from vllm_b200 import marlin_utils as mu
    L = H.make_layer(K, N, qtype, group, False, dtype)
    a = H.make_activations(M, K, dtype)
    out = G.run_gemm(ops, mu, L, a).astype(np.float64)
    assert _lib.load().b200q_device_error(1) == 0
    ref = (torch.from_numpy(a.astype(np.float64)).cuda() @ torch.from_numpy(_weights64(L)).cuda()).cpu().numpy()
    exact = mo.round_to_dtype(ref.astype(np.float32), dtype).astype(np.float64)
    # fp32 sums leave results on the wrong side of a rounding boundary where they lie within the sums' error of it:
    # an error of e (relative to the results' size) does so to about e / 2^-11 of fp16 results.  The decode kernel's
    # sums over 11008 are good to 3e-5, 6 %; weights rounded to 16 bits move results by more than half a step, 39 %.
    assert (out != exact).mean() < 0.12
    # and none by more than half a step and the sums' error (at most 6e-5 of the results' size in the decode kernel)
    half = 2.0 ** (-11 if dtype == "float16" else -8)
    assert np.all(np.abs(out - ref) <= 1.001 * half * np.abs(ref) + 2e-4 * np.sqrt(np.mean(ref ** 2)))


@pytest.mark.parametrize("M,E,K,N,qtype,group,dtype", [
    (8, 2, 512, 384, "uint8b128", 128, "float16"),    # eight rows an expert, single CTAs
    (33, 2, 576, 320, "uint8b128", 64, "bfloat16"),   # 33 rows, two groups a round, an odd number of steps
    (64, 2, 1024, 512, "uint4b8", 128, "bfloat16"),   # 64 rows: the widest single tile but one row
    (41, 2, 1024, 512, "uint4b8", 128, "float16"),    # the smallest pair tile
    (160, 2, 1024, 512, "uint4", 256, "float16"),     # the widest pair tile
    (161, 2, 1024, 768, "uint4b8", 64, "bfloat16"),   # a run in two tiles
    (350, 2, 512, 384, "uint8", 128, "bfloat16"),
    (350, 2, 768, 384, "uint8b128", 192, "float16"),  # groups for the decode kernel
])
def test_moe_keeps_group_scales_in_fp32(M, E, K, N, qtype, group, dtype):
    import torch
    from vllm_b200 import _lib, fused_moe
    from vllm_b200.scalar_type import scalar_types
    w1 = [H.make_layer(K, 2 * N, qtype, group, False, dtype, seed=e) for e in range(E)]
    w2 = [H.make_layer(N, K, qtype, group if N % group == 0 else -1, False, dtype, seed=50 + e) for e in range(E)]
    tdt = getattr(torch, dtype)
    a = G.t16(mo.round_to_dtype(0.1 * H.make_activations(M, K, dtype), dtype), dtype)
    gen = torch.Generator(device="cuda").manual_seed(M)
    ids = torch.stack([torch.randperm(E, device="cuda", generator=gen) for _ in range(M)]).to(torch.int32)
    tw = torch.rand(M, E, device="cuda", generator=gen) + 0.1
    stack = lambda ls, f: torch.stack([f(L) for L in ls])
    zeros = lambda ls: stack(ls, lambda L: G.ti32(L.marlin_zp)) if ls[0].has_zp else None
    out = fused_moe.fused_marlin_moe(
        a, stack(w1, lambda L: G.ti32(L.marlin_q)), stack(w2, lambda L: G.ti32(L.marlin_q)),
        stack(w1, lambda L: G.t16(L.marlin_s, dtype)), stack(w2, lambda L: G.t16(L.marlin_s, dtype)), tw, ids,
        getattr(scalar_types, qtype), w1_zeros=zeros(w1), w2_zeros=zeros(w2))
    torch.cuda.synchronize()
    assert _lib.load().b200q_device_error(1) == 0
    ref = torch.zeros(M, K, dtype=torch.float64, device="cuda")
    for e in range(E):   # every token meets every expert
        h = (a.double() @ torch.from_numpy(_weights64(w1[e])).cuda()).to(tdt).double()
        act = ((h[:, :N] / (1 + torch.exp(-h[:, :N]))).to(tdt).double() * h[:, N:]).to(tdt).double()
        y = (act @ torch.from_numpy(_weights64(w2[e])).cuda()) * tw.gather(1, (ids == e).int().argmax(1, keepdim=True)).double()
        ref += y.to(tdt).double()
    err = float((out.double() - ref).norm() / ref.norm())
    # The reference rounds where the layer rounds: gate, up, SiLU, activation, expert output.  The last rounding, of
    # the sum, is the layer's alone: 1.66e-3 of the result in bf16, 2.07e-4 in fp16.  A value that falls on the other
    # side of a rounding boundary on the way adds its step: up to 6 in a hundred with the sums of the decode kernel
    # (sqrt(3 x 0.06 x 12) of 2.07e-4 at each of three steps, 3.2e-4 in all), most with weights rounded to 16 bits.
    assert err < (2.3e-3 if dtype == "bfloat16" else 3.4e-4), err
