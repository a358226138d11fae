"""RWKV7 delta rule with the elementwise producers of its ``w``, ``a`` and ``b`` inputs fused in.

In an RWKV7 time-mix block three of the operator's six inputs are elementwise functions of
pre-activations that exist only to feed it -- with the input distributions of the reference's value test
(``test_script/test_rwkv7_value.py``): ``w = -exp(-1/2) * sigmoid(w_pre)``, ``kk = normalize(kk_pre)``
over the 64 channels of a head, ``a = -kk``, ``b = kk * sigmoid(a_pre)``.  Computed by separate kernels
they cost a write and a read of three ``[B, T, H, 64]`` tensors in the forward pass and as much again for
their gradients in the backward pass.  ``generalized_delta_rule_fused`` takes the pre-activations and
computes the three inputs where the operator's first kernel loads them; its backward pass returns the
gradients of the pre-activations.  ``w``, ``a`` and ``b`` are rounded to bfloat16 exactly as materialised
tensors would be, so the result equals ``generalized_delta_rule(r, w, k, v, a, b)`` bit for bit.

bfloat16 tensors ``[B, T, H, 64]`` only; ``producers`` is the unfused formula (the fallback for other
dtypes and the reference for tests).
"""
from __future__ import annotations

import math
import torch

from . import _lib, _ops
from .rwkv7 import HEAD_SIZE, generalized_delta_rule

W_SCALE = -math.exp(-0.5)


def producers(w_pre: torch.Tensor, kk_pre: torch.Tensor, a_pre: torch.Tensor):
    """``(w, a, b)`` from the pre-activations, computed in float32 and rounded to the input dtype."""
    dt = w_pre.dtype
    w = (W_SCALE * torch.sigmoid(w_pre.float())).to(dt)
    kk = torch.nn.functional.normalize(kk_pre.float(), dim=-1, eps=1e-12)
    return w, (-kk).to(dt), (kk * torch.sigmoid(a_pre.float())).to(dt)


def _check_args(r, w_pre, k, v, kk_pre, a_pre, initial_state):
    """Raise what the interface documents for invalid arguments (the operator itself only says that they are)."""
    _lib.require_cuda(r, w_pre, k, v, kk_pre, a_pre, initial_state)
    if r.dim() != 4 or r.shape[-1] != HEAD_SIZE:
        raise ValueError(f"expected 4-D token tensors with head size {HEAD_SIZE}, got {tuple(r.shape)}")
    for name, x in (("w_pre", w_pre), ("k", k), ("v", v), ("kk_pre", kk_pre), ("a_pre", a_pre)):
        if x.shape != r.shape:
            raise ValueError(f"{name} has shape {tuple(x.shape)}, expected {tuple(r.shape)}")
    B, H = r.shape[0], r.shape[2]
    if initial_state is not None and (initial_state.dim() != 4 or initial_state.shape[0] not in (1, B)
                                      or tuple(initial_state.shape[1:]) != (H, HEAD_SIZE, HEAD_SIZE)):
        raise ValueError(
            f"initial_state must be [{B} or 1, {H}, {HEAD_SIZE}, {HEAD_SIZE}], got {tuple(initial_state.shape)}")


def generalized_delta_rule_fused(r, w_pre, k, v, kk_pre, a_pre, initial_state=None, output_final_state=True):
    """``generalized_delta_rule(r, w, k, v, a, b)`` with ``(w, a, b) = producers(w_pre, kk_pre, a_pre)``
    computed inside the operator (see the module docstring).  ``[B, T, H, 64]`` tensors; returns
    ``(o, final_state)`` or just ``o``."""
    try:
        if r.dtype == torch.bfloat16 and r.dim() == 4 and r.shape[1] > 1 and w_pre.dtype == k.dtype == v.dtype \
                == kk_pre.dtype == a_pre.dtype == torch.bfloat16:
            o, ht = _ops.load().rwkv7_fused(r, w_pre, k, v, kk_pre, a_pre, initial_state)
            return (o, ht) if output_final_state else o
    except Exception as e:
        _check_args(r, w_pre, k, v, kk_pre, a_pre, initial_state)
        raise _ops.failed(e)
    _check_args(r, w_pre, k, v, kk_pre, a_pre, initial_state)
    w, a, b = producers(w_pre, kk_pre, a_pre)      # unfused: other dtypes and single-token steps
    return generalized_delta_rule(r, w, k, v, a, b, initial_state=initial_state, output_final_state=output_final_state)
