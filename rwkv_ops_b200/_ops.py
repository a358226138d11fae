"""The torch operators of ``csrc/torch_ops.cpp``, loaded once, and their shape functions.

``load()`` returns the operator namespace (``torch.ops.rwkv_ops_b200``); it raises if one of the two libraries has
not been built.  ``failed(error)`` turns an operator's error into the exception the package documents.
"""
from __future__ import annotations

import os

import torch

from . import _lib
from ._lib import RwkvB200Error

OPS_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "librwkv_ops_b200_torch.so")

_ops = None


def load():
    global _ops
    if _ops is None:
        _lib.load()      # the C ABI the operators call
        if not os.path.exists(OPS_PATH):
            raise RwkvB200Error(f"{OPS_PATH} not found. Build it with `python -m rwkv_ops_b200.build`; "
                                     "rwkv_ops_b200 has no eager fallback.")
        try:
            torch.ops.load_library(OPS_PATH)
        except OSError as e:
            raise RwkvB200Error(f"{OPS_PATH} does not load with torch {torch.__version__}; rebuild it with "
                                f"`python -m rwkv_ops_b200.build`: {e}") from e
        _register_fakes()
        _ops = torch.ops.rwkv_ops_b200
    return _ops


def built() -> bool:
    return os.path.exists(OPS_PATH) and os.path.exists(_lib.LIB_PATH)


def failed(error: Exception) -> Exception:
    """What to raise for an operator call that failed on valid arguments."""
    text = str(error)
    if type(error) is RuntimeError and text.startswith("rwkv_ops_b200 "):
        return RwkvB200Error(text.splitlines()[0])
    return error


def _register_fakes():
    fake = torch.library.register_fake

    def state(r, n, H, K):
        return r.new_empty((n, H, K, K), dtype=torch.float32)

    def tokens(r, n):
        return tuple(torch.empty_like(r) for _ in range(n))

    def kept(r, n):
        return r.new_empty((n,), dtype=torch.uint8)

    def dims(r, head_first):
        B, T, H, K = r.shape
        return (B, H, T, K) if head_first else (B, T, H, K)

    @fake("rwkv_ops_b200::rwkv7_fwd")
    def _(r, w, k, v, a, b, h0, head_first, algo, keep):
        B, T, H, K = dims(r, head_first)
        tiles = K == 64 and r.dtype == torch.bfloat16 and algo & 0xff != _lib.ALGO_RECURRENT
        n = 0 if not keep else _lib.rwkv7_kept_bytes(B, T, H) if tiles else _lib.rwkv7_states_bytes(B, T, H, K)
        return torch.empty_like(r), state(r, B, H, K), kept(r, n)

    @fake("rwkv_ops_b200::rwkv7_bwd")
    def _(r, w, k, v, a, b, h0, d_o, d_ht, k_, head_first, algo):
        B, T, H, K = dims(r, head_first)
        return (*tokens(r, 6), state(r, B, H, K))

    @fake("rwkv_ops_b200::rwkv7_decode_step")
    def _(r, w, k, v, a, b, state):
        return torch.empty_like(r)

    @fake("rwkv_ops_b200::rwkv7_fwd_varlen")
    def _(r, w, k, v, a, b, seq_start, seq_len, max_len, h0, keep):
        H, n = r.shape[2], seq_start.numel()
        return torch.empty_like(r), state(r, n, H, 64), kept(r, _lib.rwkv7_kept_bytes(n, max_len, H) if keep else 0)

    @fake("rwkv_ops_b200::rwkv7_bwd_varlen")
    def _(r, w, k, v, a, b, seq_start, seq_len, max_len, h0, d_o, d_ht, k_):
        return (*tokens(r, 6), state(r, seq_start.numel(), r.shape[2], 64))

    @fake("rwkv_ops_b200::rwkv7_fused_fwd")
    def _(r, w_pre, k, v, kk_pre, a_pre, h0, keep):
        B, T, H, K = r.shape
        return torch.empty_like(r), state(r, B, H, K), kept(r, _lib.rwkv7_kept_bytes(B, T, H) if keep else 0)

    @fake("rwkv_ops_b200::rwkv7_fused_bwd")
    def _(r, w_pre, k, v, kk_pre, a_pre, h0, d_o, d_ht, k_):
        B, T, H, K = r.shape
        return (*tokens(r, 6), state(r, B, H, K))

    @fake("rwkv_ops_b200::wkv6_fwd")
    def _(r, k, v, w, u, s0, state_map, algo, keep):
        B, T, C = r.shape
        H, N = u.shape
        sT = state(r, B, H, N)
        return (torch.empty_like(r), sT.to(r.dtype) if algo & _lib.ALGO_TOKEN_STATES else sT,
                kept(r, _lib.wkv6_kept_bytes(B, T, H) if keep else 0))

    @fake("rwkv_ops_b200::wkv6_bwd")
    def _(r, k, v, w, u, s0, state_map, d_y, d_sT, k_, algo):
        return (*tokens(r, 4), torch.empty_like(u), state(r, r.shape[0], *u.shape))

    @fake("rwkv_ops_b200::wkv6_fwd_varlen")
    def _(r, k, v, w, u, seq_start, seq_len, max_len, s0, state_map, keep):
        H, N = u.shape
        n = seq_start.numel()
        return torch.empty_like(r), state(r, n, H, N), kept(r, _lib.wkv6_kept_bytes(n, max_len, H) if keep else 0)

    @fake("rwkv_ops_b200::wkv6_bwd_varlen")
    def _(r, k, v, w, u, seq_start, seq_len, max_len, s0, state_map, d_y, d_sT, k_):
        return (*tokens(r, 4), torch.empty_like(u), state(r, seq_start.numel(), *u.shape))
