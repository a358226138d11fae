"""Tracing without a device: the operators on fake CUDA tensors whose batch and length are symbols keep them symbols (a
program traced once serves every length), and an exported program takes a dynamic length."""
import pytest
import torch
from torch._dynamo.source import ConstantSource
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.symbolic_shapes import DimDynamic, ShapeEnv
from torch.utils._python_dispatch import TorchDispatchMode

import rwkv_ops_b200 as ro
from rwkv_ops_b200 import _ops
from rwkv_ops_b200.build import build


@pytest.fixture(scope="module", autouse=True)
def _operators():
    if not _ops.built():
        build()
    _ops.load()


def _tokens(n, shape, dtype=torch.bfloat16):
    """``n`` fake tensors of ``shape`` whose first two dimensions are symbols."""
    env = ShapeEnv()
    mode = FakeTensorMode(shape_env=env)
    sizes = list(shape)
    for i in (0, 1):
        src = ConstantSource(f"size{i}")
        sizes[i] = env.create_symintnode(env.create_symbol(shape[i], src, DimDynamic.DYNAMIC), hint=shape[i], source=src)
    with mode:
        return mode, sizes, [torch.empty(sizes, dtype=dtype, device="cuda") for _ in range(n)]


def _symbolic(t, dims):
    return [isinstance(t.shape[i].node.maybe_as_int() if isinstance(t.shape[i], torch.SymInt) else t.shape[i], type(None)) for i in dims]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rwkv7_keeps_symbolic_sizes(dtype):
    mode, sizes, x = _tokens(6, (2, 100, 3, 64), dtype)
    with mode, torch.no_grad():
        for state in (None, torch.empty(1, 3, 64, 64, device="cuda"), torch.empty(sizes[0], 3, 64, 64, device="cuda")):
            o, s = ro.generalized_delta_rule(*x, initial_state=state)
            assert all(_symbolic(o, (0, 1))) and all(_symbolic(s, (0,)))
        if dtype == torch.bfloat16:
            o, s = ro.generalized_delta_rule_fused(*x)
            assert all(_symbolic(o, (0, 1))) and all(_symbolic(s, (0,)))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_wkv6_keeps_symbolic_sizes(dtype):
    mode, sizes, x = _tokens(4, (2, 100, 128), dtype)
    with mode, torch.no_grad():
        u = torch.empty(2, 64, dtype=dtype, device="cuda")
        table = torch.empty(3, 2, 64, 64, dtype=dtype, device="cuda")
        state_map = torch.empty(sizes[0], dtype=torch.int64, device="cuda")
        for kw in ({}, dict(init_state=table[:1]), dict(init_state=table, state_map=state_map)):
            y, s = ro.RWKV6_OP(64, 100)(*x, u, with_state=True, **kw)
            assert all(_symbolic(y, (0, 1))) and all(_symbolic(s, (0,)))


def test_wkv6_training_keeps_symbolic_sizes():
    mode, sizes, x = _tokens(4, (2, 100, 128))
    with mode:
        u = torch.empty(2, 64, dtype=torch.bfloat16, device="cuda")
        x[0].requires_grad_(True)
        y, s = ro.RWKV6_OP(64, 100)(*x, u, with_state=True)
        assert y.requires_grad and all(_symbolic(y, (0, 1))) and all(_symbolic(s, (0,)))


def test_float32_rwkv7_training_keeps_symbolic_sizes():
    mode, sizes, x = _tokens(6, (2, 100, 3, 64), torch.float32)
    with mode:
        x[0].requires_grad_(True)
        o, s = ro.generalized_delta_rule(*x)
        assert o.requires_grad and all(_symbolic(o, (0, 1))) and all(_symbolic(s, (0,)))


class Layer(torch.nn.Module):
    def forward(self, *x):
        o, s = ro.generalized_delta_rule(*x)
        return 2 * o, s


def test_export_with_a_dynamic_length():
    length = torch.export.Dim("length", min=2, max=8192)
    with FakeTensorMode(shape_env=ShapeEnv()), torch.no_grad():
        x = tuple(torch.empty(2, 100, 3, 64, dtype=torch.bfloat16, device="cuda") for _ in range(6))
        program = torch.export.export(Layer(), x, dynamic_shapes=(tuple({1: length} for _ in x),))
    assert any("rwkv_ops_b200" in str(n.target) for n in program.graph.nodes)


@pytest.mark.parametrize("longest", [8192, None])
@pytest.mark.parametrize("traced", [8, 16, 17, 100])
@pytest.mark.parametrize("dtype,K", [(torch.float32, 64), (torch.float32, 128), (torch.float16, 64), (torch.bfloat16, 128)])
def test_export_of_the_float32_recurrence_with_gradients(dtype, K, traced, longest):
    """Whatever length it is traced at, the program serves all that were declared, on either side of 16 tokens, from which on the
    forward leaves states for its backward, and without a bound from the memory these may take."""
    length = torch.export.Dim("length", min=2, max=longest)
    with FakeTensorMode(shape_env=ShapeEnv()):
        x = tuple(torch.empty(2, traced, 3, K, dtype=dtype, device="cuda", requires_grad=True) for _ in range(6))
        program = torch.export.export(Layer(), x, dynamic_shapes=(tuple({1: length} for _ in x),))
    (bounds,) = program.range_constraints.values()
    assert bounds.lower == 2 and (longest is None or bounds.upper == longest)


class _Calls(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.keep = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if func is torch.ops.rwkv_ops_b200.rwkv7_fwd.default:
            self.keep.append(args[-1])
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("T,limit,keep", [(8, None, False), (16, None, False), (17, None, True), (100, None, True), (100, "0", False)])
def test_states_are_kept_by_length_and_limit(T, limit, keep, monkeypatch):
    if limit is not None:
        monkeypatch.setenv("RWKV_OPS_B200_KEEP_LIMIT_MB", limit)
    with FakeTensorMode():
        x = [torch.empty(2, T, 3, 64, device="cuda", requires_grad=True) for _ in range(6)]
        with _Calls() as calls:
            ro.generalized_delta_rule(*x)
    assert calls.keep == [keep]


def test_wrong_arguments_still_raise():
    mode, sizes, x = _tokens(6, (2, 100, 3, 64))
    with mode, torch.no_grad():
        with pytest.raises(ValueError):
            ro.generalized_delta_rule(*x[:5], x[5][:, :-1])
        with pytest.raises(ValueError):
            ro.generalized_delta_rule(*x, initial_state=torch.empty(3, 3, 64, 64, device="cuda"))
        with pytest.raises(ValueError):
            ro.generalized_delta_rule(*[t[..., :32] for t in x])
