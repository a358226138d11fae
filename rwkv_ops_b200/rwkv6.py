"""RWKV6 wkv operator: the reference's ``RWKVKernelOperator`` interface over the CUDA library.

Mirrors ``get_rwkv6_kernel`` / ``RWKVKernelOperator`` of the reference
(``rwkv_ops/rwkv6_kernel/__init__.py:9-96``, ``rwkv_ops/rwkv6_kernel/ops_rwkv_kernel.py:5-86``,
``rwkv_ops/rwkv6_kernel/torch_rwkv_kernel.py:50-304``): constructor ``(head_size,
max_sequence_length, ops_loop=False)`` and call ``(r, k, v, w, u, with_state=False,
init_state=None, state_map=None) -> (y, state | None)``.  Unlike the reference's GPU operator,
gradients flow with ``with_state=True`` (to ``init_state`` as well), ``state_map`` works, and
``max_sequence_length`` is not a compile-time constant (it is accepted and ignored).
"""
from __future__ import annotations

import os

import torch

from . import _lib, _ops

HEAD_SIZE = 64                  # the head size of the chunked tensor-core path
HEAD_SIZES = (32, 64, 128)      # 32 and 128 run the float32 recurrence
_ALGO_NAMES = {"auto": _lib.ALGO_AUTO, "recurrent": _lib.ALGO_RECURRENT, "chunked": _lib.ALGO_CHUNKED}


def _default_algo() -> int:
    return _ALGO_NAMES[os.environ.get("RWKV_OPS_B200_WKV6_ALGO", "auto").lower()]


class RWKVKernelOperator:
    """Drop-in for the class returned by the reference's ``get_rwkv6_kernel``."""

    def __init__(self, head_size, max_sequence_length, ops_loop=False):
        if head_size not in HEAD_SIZES:
            raise ValueError(f"rwkv_ops_b200 wkv6 supports head sizes {HEAD_SIZES}, got {head_size}")
        self.head_size = head_size
        self.max_sequence_length = max_sequence_length   # kept for compatibility; no limit applies
        self.ops_loop = ops_loop

    def _check_args(self, r, k, v, w, u, init_state, state_map):
        """Raise what the interface documents for invalid arguments (the operator itself only says that they are)."""
        _lib.require_cuda(r, k, v, w, u, init_state)
        if r.dim() != 3:
            raise ValueError(f"expected [B, T, C] tensors, got {tuple(r.shape)}")
        B, T, C = r.shape
        N = self.head_size
        assert C % N == 0, "hidden size must be a multiple of head_size"
        H = C // N
        for name, x in (("k", k), ("v", v), ("w", w)):
            assert x.shape == r.shape, f"{name} has shape {tuple(x.shape)}, expected {tuple(r.shape)}"
            assert x.dtype == r.dtype, "r, k, v, w must share one dtype"
        assert u.numel() == C, f"u must have {C} elements"
        if init_state is not None:
            assert init_state.dim() in (3, 4), "init_state must be [n_state, H, N, N] or [H, N, N]"
            assert tuple(init_state.shape[-3:]) == (H, N, N), "init_state must be [n_state, H, N, N] or [H, N, N]"
            n_state = 1 if init_state.dim() == 3 else init_state.shape[0]
            if state_map is None:
                if n_state not in (1, B):
                    raise ValueError("state_map cannot be inferred from init_state; pass it explicitly")
            else:
                assert state_map.dtype in (torch.int32, torch.int64), "state_map must be int32 or int64"
                assert state_map.numel() == B, "state_map must have one entry per batch row"
        else:
            assert state_map is None, "state_map needs init_state"
        if N != HEAD_SIZE and _default_algo() == _lib.ALGO_CHUNKED:
            raise ValueError("the chunked wkv6 path is built for head size 64")

    def __call__(self, r, k, v, w, u, with_state=False, init_state=None, state_map=None):
        host_map = state_map
        try:
            if state_map is not None and not (isinstance(state_map, torch.Tensor) and state_map.is_cuda):
                if isinstance(state_map, (list, tuple)):
                    host_map = state_map = torch.tensor(state_map, dtype=torch.int32)
                assert init_state is not None, "state_map needs init_state"
                # a host-side map (list, CPU tensor) is range-checked here, where the reference
                # device-asserts (rwkv6_kernel/torch_kernel/wkv6_cuda.cu:81); a map that already lives
                # on the device is not read back (that would stall the stream on every call): the
                # kernels clamp its entries to the table instead of trapping
                n_state = 1 if init_state.dim() == 3 else init_state.shape[0]
                assert bool((state_map >= 0).all()) and bool((state_map < n_state).all()), (
                    f"state_map values must lie in [0, {n_state})")
                state_map = state_map.to(r.device)
            y, sT = _ops.load().wkv6(r, k, v, w, u, self.head_size, init_state, state_map, bool(with_state))
        except Exception as e:
            self._check_args(r, k, v, w, u, init_state, host_map)
            raise _ops.failed(e)
        return y, sT if with_state else None


def get_rwkv6_kernel(KERNEL_TYPE: str = "cuda"):
    """Reference signature (``rwkv_ops/rwkv6_kernel/__init__.py:9``); ``KERNEL_TYPE`` is ignored."""
    return RWKVKernelOperator
