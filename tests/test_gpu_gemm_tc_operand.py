"""Where the tensor-core kernel keeps its converted weights: in TMEM up to 192 tokens a tile (four, three or two rounds
of them, by the tile's width), in shared memory above.  The widths at which that changes, for single CTAs and, with enough
columns, CTA pairs; an odd number of steps, a last column tile of 64, several scale groups within a step and groups that
begin anywhere in one."""
import pytest

from oracle import marlin_oracle as mo
from tests import helpers as H

pytestmark = pytest.mark.gpu
WIDE = 148 * 128 + 64   # more column tiles than SMs


@pytest.mark.parametrize("M,K,N,qtype,group,dtype", [
    (33, 192, 192, "uint4b8", 32, "bfloat16"),
    (64, 320, 320, "uint8", 64, "bfloat16"),
    (65, 192, 192, "uint8b128", 96, "bfloat16"),
    (128, 576, 320, "uint4", 192, "float16"),
    (100, 192, WIDE, "uint4b8", 96, "float16"),
    (128, 192, WIDE, "uint8", 32, "bfloat16"),
    (129, 192, WIDE, "uint4", 64, "bfloat16"),
    (160, 320, WIDE, "uint8b128", -1, "float16"),
    (161, 192, WIDE, "uint4b8", 32, "float16"),
    (192, 320, WIDE, "uint8", 64, "float16"),
    (193, 192, WIDE, "uint4", 32, "bfloat16"),
    (193, 192, WIDE, "uint8", 96, "bfloat16"),
    (256, 320, WIDE, "uint8b128", 64, "bfloat16"),
    (640, 192, WIDE, "uint4b8", 64, "bfloat16"),
])
def test_operand_places(M, K, N, qtype, group, dtype):
    from tests import gpu_utils as G
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import _lib
    from vllm_b200 import marlin_utils as mu
    L = H.make_layer(K, N, qtype, group, False, dtype, with_bias=M % 2 == 1)
    a = H.make_activations(M, K, dtype)
    out = G.run_gemm(ops, mu, L, a)
    assert _lib.load().b200q_device_error(1) == 0
    max_frac, mean_rel = H.gemm_errors(out, mo.gemm_ref(a, L.w, L.bias))
    assert max_frac <= H.MAX_ABS_FRAC and mean_rel <= H.MEAN_REL, (max_frac, mean_rel)
