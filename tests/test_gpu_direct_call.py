"""The direct call (the GEMM operator without the dispatcher) steps aside, by returning None, wherever something wants
to see operators, and gives the operator's bits everywhere else."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def call():
    import torch
    from vllm_b200 import _custom_ops as ops
    from vllm_b200 import marlin_utils as mu
    from vllm_b200.scalar_type import scalar_types
    K, N = 1024, 512
    gen = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randint(-2**31, 2**31 - 1, (K // 16, N * 2), dtype=torch.int32, device="cuda", generator=gen)
    s = (torch.rand((K // 128, N), device="cuda", generator=gen) * 0.018 + 0.002).half()
    e = torch.empty(0, dtype=torch.int32, device="cuda")
    ws = mu.marlin_make_workspace_new(torch.device("cuda"))
    x = torch.randn((3, 5, K), device="cuda", dtype=torch.float16, generator=gen)

    def make(x=x, bias=None, s=s, through=ops._linear):
        if through is ops._linear:
            return ops._linear(x, q, bias, s, None, e, e, e, ws, scalar_types.uint4b8.id, -1, N, K, ops.K_FULL)
        return ops.linear(x, q, bias, s, None, e, e, e, ws, scalar_types.uint4b8.id, N, K)

    make.x, make.s, make.ops = x, s, ops
    a = x.reshape(-1, K)
    make.operator = getattr(torch.ops, ops.ops_namespace()).gptq_marlin_gemm(
        a, None, q, None, s, None, e, e, e, ws, scalar_types.uint4b8.id, a.shape[0], N, K, True, False, True,
        False).reshape(3, 5, N)
    return make


def test_direct_call_gives_the_operators_bits(call):
    import torch
    direct = call()
    assert direct is not None and direct.shape == call.operator.shape and torch.equal(direct, call.operator)
    with torch.no_grad():
        assert torch.equal(call(call.x.clone().requires_grad_()), call.operator)
    strided = torch.empty((3, 5, 2048), device="cuda", dtype=torch.float16)[..., :1024]
    strided.copy_(call.x)
    assert torch.equal(call(strided), call.operator)


def _modes():
    import torch
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    return {"dispatch mode": Dispatch, "function mode": Function, "inference mode": torch.inference_mode,
            "profiler": torch.profiler.profile}


@pytest.mark.parametrize("mode", ["dispatch mode", "function mode", "inference mode", "profiler"])
def test_direct_call_steps_aside_in(call, mode):
    import torch
    with _modes()[mode]():
        assert call() is None
        out = call(through=call.ops.linear)
    assert torch.equal(out, call.operator)
    assert call() is not None


def test_direct_call_steps_aside_for_subclasses_and_autograd(call):
    import torch

    class Sub(torch.Tensor):
        pass

    assert call(call.x.as_subclass(Sub)) is None
    assert isinstance(call(call.x.as_subclass(Sub), through=call.ops.linear), Sub)
    assert call(call.x.clone().requires_grad_()) is None
    assert call(s=call.s.clone().requires_grad_()) is None
    assert call(bias=torch.zeros(512, device="cuda", dtype=torch.float16).requires_grad_()) is None
    assert call(bias=torch.nn.Parameter(torch.zeros(512, device="cuda", dtype=torch.float16), requires_grad=False)) is not None


def test_direct_call_steps_aside_under_vmap_and_tracing(call):
    import torch
    seen = []

    def body(x):
        seen.append(call(x))
        return x + 1

    torch.vmap(body)(call.x)
    torch.func.grad(lambda x: body(x).sum())(call.x.float())
    torch.jit.trace(body, (call.x,), check_trace=False)
    assert seen == [None] * 3
