"""RWKV7 generalized delta rule: the reference's Python interface over the CUDA library.

Mirrors ``generalized_delta_rule`` and ``get_generalized_delta_rule`` of the reference
(``rwkv_ops/rwkv7_kernel/native_keras_op.py:23-95``, ``rwkv_ops/rwkv7_kernel/torch_op.py:458-490``,
``rwkv_ops/rwkv7_kernel/__init__.py:14-156``): same argument names and meaning, ``exp(-exp(w))``
decay, output in ``r``'s dtype, float32 states in the native ``[N, H, V, K]`` layout, a bare
tensor when ``output_final_state`` is false.  The work is done by torch operators with autograd
(``csrc/torch_ops.cpp``) that call the C ABI; there is no Triton, no multi-backend dispatch
and no CPU fallback.
"""
from __future__ import annotations

import os
from typing import Optional

import torch

from . import _lib, _ops

HEAD_SIZE = 64               # the head size of the tensor-core path
HEAD_SIZES = (64, 128)       # head sizes the operator accepts (128: float32 recurrence for every dtype)
_ALGO_NAMES = {"auto": _lib.ALGO_AUTO, "recurrent": _lib.ALGO_RECURRENT, "chunked": _lib.ALGO_CHUNKED}


def _default_algo() -> int:
    return _ALGO_NAMES[os.environ.get("RWKV_OPS_B200_RWKV7_ALGO", "auto").lower()]


def _check_args(r, w, k, v, a, b, initial_state, head_first):
    """Raise what the interface documents for invalid arguments (the operator itself only says that they are)."""
    _lib.require_cuda(r, w, k, v, a, b, initial_state)
    if r.dim() != 4 or r.shape[-1] not in HEAD_SIZES:
        raise ValueError(f"expected 4-D token tensors with head size in {HEAD_SIZES}, got {tuple(r.shape)}")
    for name, x in (("w", w), ("k", k), ("v", v), ("a", a), ("b", b)):
        if x.shape != r.shape:
            raise ValueError(f"{name} has shape {tuple(x.shape)}, expected {tuple(r.shape)}")
    B, N = r.shape[0], r.shape[-1]
    H = r.shape[1] if head_first else r.shape[2]
    if initial_state is not None:
        if initial_state.dim() != 4 or tuple(initial_state.shape[1:]) != (H, N, N) \
                or initial_state.shape[0] not in (1, B):
            raise ValueError(f"initial_state must be [{B} or 1, {H}, {N}, {N}], got {tuple(initial_state.shape)}")
    _default_algo()


def generalized_delta_rule(
    r: torch.Tensor,
    w: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    a: torch.Tensor,
    b: torch.Tensor,
    initial_state: Optional[torch.Tensor] = None,
    output_final_state: bool = True,
    head_first: bool = False,
):
    """Drop-in for the reference's ``generalized_delta_rule``.

    ``r, w, k, v, a, b``: ``[B, T, H, K]`` (``[B, H, T, K]`` when ``head_first``) with head size
    ``K`` 64 or 128 (the reference's value test runs 128, ``test_script/test_rwkv7_value.py:46-51``), any
    of float32 / bfloat16 / float16; ``w`` is the raw decay input (the operator applies
    ``exp(-exp(w))``).  ``initial_state``: float32 ``[N, H, K, K]`` with ``N == B`` or ``N == 1``
    (broadcast), value index before key index.  Returns ``(o, final_state)`` or just ``o``.
    Head size 64 with bfloat16 tokens takes the tensor-core path, everything else the float32 recurrence
    (``RWKV_OPS_B200_RWKV7_ALGO=chunked`` sends float32 / float16 tokens of head size 64 through the tensor-core
    path as well, rounded to bfloat16).
    """
    try:
        o, ht = _ops.load().generalized_delta_rule(r, w, k, v, a, b, initial_state, bool(head_first))
    except Exception as e:
        _check_args(r, w, k, v, a, b, initial_state, head_first)
        raise _ops.failed(e)
    return (o, ht) if output_final_state else o


def get_generalized_delta_rule(HEAD_SIZE: int = 64, KERNEL_TYPE: str = "cuda"):
    """Reference signature (``rwkv_ops/rwkv7_kernel/__init__.py:14``): returns ``(fn, USE_KERNEL)``.

    ``USE_KERNEL`` is always True (callers use it to choose the padding recipe of the kernel
    path).  ``KERNEL_TYPE`` is accepted for compatibility and ignored: there is one implementation.
    """
    if HEAD_SIZE not in HEAD_SIZES:
        raise ValueError(f"rwkv_ops_b200 is built for head sizes {HEAD_SIZES}")
    return generalized_delta_rule, True
