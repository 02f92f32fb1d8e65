"""The last token tile of the tensor-core kernel runs its MMAs only as wide as its rows: last tiles of one row, of a row
beyond a step of 16 (pairs 32) and of nearly the whole width, in single CTAs and pairs, weights in TMEM and in shared memory,
the last column tile half a tile.  And the calls on both sides of the lines between the decode and the tensor-core kernel."""
import pytest

from oracle import marlin_oracle as mo
from tests import helpers as H
from tests import test_gpu_group_sums as sums

pytestmark = pytest.mark.gpu
WIDE = 148 * 128 + 64   # more column tiles than SMs


@pytest.mark.parametrize("M,K,N,qtype,group,dtype", [
    (257, 192, 320, "uint4b8", 64, "bfloat16"),       # single CTAs, tiles of 64, the last of one row
    (145, 320, 320, "uint8", 64, "float16"),          # 17 rows
    (513, 192, 320, "uint8b128", -1, "float16"),      # pairs, tiles of 128, the last of one row
    (449, 192, 320, "uint4", 64, "bfloat16"),         # 65 rows
    (2049, 128, 1024, "uint4b8", -1, "float16"),      # single CTAs, tiles of 128, one row
    (4097, 128, 1024, "uint4b8", 32, "bfloat16"),     # pairs, tiles of 256, one row
    (4129, 128, 1024, "uint8b128", 64, "float16"),    # 33 rows
    (290, 128, WIDE, "uint4b8", 64, "bfloat16"),      # pairs, tiles of 160, 130 rows
    (353, 128, WIDE, "uint8", 32, "float16"),         # pairs, tiles of 192, 161 rows
])
def test_last_tile(M, K, N, qtype, group, dtype):
    from tests import gpu_utils as G
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import _lib
    from vllm_b200 import marlin_utils as mu
    L = H.make_layer(K, N, qtype, group, False, dtype, with_bias=M % 2 == 1)
    a = H.make_activations(M, K, dtype)
    out = G.run_gemm(ops, mu, L, a)
    assert _lib.load().b200q_device_error(1) == 0
    ref = mo.gemm_ref(a, L.w, L.bias)
    for part in (slice(None), slice(M - M % 32, None) if M % 32 else slice(-32, None)):
        max_frac, mean_rel = H.gemm_errors(out[part], ref[part])
        assert max_frac <= H.MAX_ABS_FRAC and mean_rel <= H.MEAN_REL, (max_frac, mean_rel)


@pytest.mark.parametrize("M,K,N,qtype,group,dtype", [
    (16, 14336, 4096, "uint4b8", 64, "bfloat16"),     # decode kernel
    (17, 14336, 4096, "uint4b8", 64, "bfloat16"),     # tensor cores
    (20, 3584, 4608, "uint4b8", 64, "bfloat16"),
    (32, 2048, 2048, "uint4b8", 128, "bfloat16"),
])
def test_few_rows_at_the_line(M, K, N, qtype, group, dtype):
    sums.test_few_rows_keep_group_scales_in_fp32(M, K, N, qtype, group, dtype)


@pytest.mark.parametrize("M,group,qtype", [(14, 64, "uint4b8"), (15, 64, "uint4b8"), (13, 128, "uint4b8"), (14, 128, "uint4b8"),
                                           (13, 64, "uint8b128"), (14, 64, "uint4"), (1, 128, "uint8b128"), (2, 128, "uint8b128")])
def test_expert_layers_at_the_line(M, group, qtype):
    sums.test_moe_keeps_group_scales_in_fp32(M, 2, 512, 384, qtype, group, "bfloat16")
