"""RWKV7 generalized delta rule on packed variable-length batches.

The reference carries ``cu_seqlens`` plumbing for this in its Triton path but has it disabled
(``rwkv_ops/rwkv7_kernel/torch_op.py:283,299``, the ``if False:`` blocks of e.g.
``triton_kernel/chunk_A_fwd.py:47-56``); its users pad every sequence to the longest one and push the
padding's decay input to ``-1e9`` (``README.md:92-98``).  ``generalized_delta_rule_varlen`` takes the
sequences laid end to end instead -- token tensors ``[1, total_len, H, 64]`` plus ``cu_seqlens``
``[n_seq + 1]`` (``cu_seqlens[i]`` is the first token of sequence ``i``) -- and returns what running the
operator on every sequence alone would: ``o`` ``[1, total_len, H, 64]`` and one final state per
sequence ``[n_seq, H, 64, 64]``.  No padded token is ever loaded or stored.

bfloat16 token tensors run on the chunked tensor-core kernels (chunk slots past the end of a sequence
are skipped, a partial last chunk is stored row by row so that the next sequence's rows stay intact);
other dtypes run the dense operator once per sequence.
"""
from __future__ import annotations

import torch

from . import _lib, _ops
from .rwkv7 import HEAD_SIZE, generalized_delta_rule


def _seq_arrays(cu_seqlens, total_len: int, device):
    cu = torch.as_tensor(cu_seqlens).detach().to("cpu", torch.int64).flatten()
    if cu.numel() < 2 or int(cu[0]) != 0 or int(cu[-1]) != total_len:
        raise ValueError(f"cu_seqlens must run from 0 to the number of tokens ({total_len}), got {cu.tolist()}")
    lens = cu[1:] - cu[:-1]
    if int(lens.min()) < 1:
        raise ValueError("every sequence must hold at least one token")
    start = cu[:-1].to(device=device, dtype=torch.int32)
    return cu, start, lens.to(device=device, dtype=torch.int32), int(lens.max())


class PackedSequences:
    """``cu_seqlens`` prepared once (host copy, device arrays of first tokens and lengths, longest length)
    for all the calls that share it, e.g. every layer of a step; pass it in place of ``cu_seqlens``."""

    def __init__(self, cu_seqlens, device="cuda"):
        cu = torch.as_tensor(cu_seqlens).detach().to("cpu", torch.int64).flatten()
        self.total_len = int(cu[-1]) if cu.numel() else 0
        self.device = torch.device(device)
        self.cu, self.start, self.lens, self.max_len = _seq_arrays(cu, self.total_len, self.device)


def _pack(cu_seqlens, total_len, device):
    """A ``PackedSequences`` for one call; ``cu_seqlens`` must end at ``total_len``."""
    p = PackedSequences.__new__(PackedSequences)
    p.total_len, p.device = total_len, device
    p.cu, p.start, p.lens, p.max_len = _seq_arrays(cu_seqlens, total_len, device)
    return p


def _token_args(r, w, k, v, a, b):
    """The six token tensors in ``r``'s dtype, contiguous: the kernels read all of them as one element type
    (``generalized_delta_rule`` casts in the same way; under mixed precision ``w`` often arrives as float32)."""
    return [x.to(r.dtype).contiguous() for x in (r, w, k, v, a, b)]


def _check_args(r, w, k, v, a, b, initial_state, cu_seqlens):
    """Raise what the interface documents for invalid arguments (the operator itself only says that they are)."""
    dev = _lib.require_cuda(r, w, k, v, a, b, initial_state)
    if r.dim() != 4 or r.shape[0] != 1 or r.shape[-1] != HEAD_SIZE:
        raise ValueError(f"expected packed token tensors [1, total_len, H, {HEAD_SIZE}], got {tuple(r.shape)}")
    for name, x in (("w", w), ("k", k), ("v", v), ("a", a), ("b", b)):
        if x.shape != r.shape:
            raise ValueError(f"{name} has shape {tuple(x.shape)}, expected {tuple(r.shape)}")
    if isinstance(cu_seqlens, PackedSequences) and (cu_seqlens.total_len != r.shape[1] or cu_seqlens.start.device != dev):
        raise ValueError("the PackedSequences object was made for another token count or device")
    H = r.shape[2]
    if initial_state is not None and (initial_state.dim() != 4
                                      or tuple(initial_state.shape[1:]) != (H, HEAD_SIZE, HEAD_SIZE)):
        raise ValueError(f"initial_state must be [n_seq or 1, {H}, {HEAD_SIZE}, {HEAD_SIZE}], "
                         f"got {tuple(initial_state.shape)}")


def generalized_delta_rule_varlen(r, w, k, v, a, b, cu_seqlens, initial_state=None, output_final_state=True):
    """``generalized_delta_rule`` over sequences packed end to end (see the module docstring).

    ``r, w, k, v, a, b``: ``[1, total_len, H, 64]``; ``cu_seqlens``: ``n_seq + 1`` increasing integers from
    0 to ``total_len`` (tensor or list, or a ``PackedSequences`` made from them once); ``initial_state``: float32 ``[n_seq or 1, H, 64, 64]``.
    Returns ``(o, final_state)`` with ``final_state`` ``[n_seq, H, 64, 64]``, or just ``o``.
    """
    try:
        if isinstance(cu_seqlens, PackedSequences) and r.dtype == torch.bfloat16 \
                and cu_seqlens.total_len == r.shape[1] and cu_seqlens.start.device == r.device:
            p = cu_seqlens
        else:
            _check_args(r, w, k, v, a, b, initial_state, cu_seqlens)
            p = cu_seqlens if isinstance(cu_seqlens, PackedSequences) else _pack(cu_seqlens, r.shape[1], r.device)
        if r.dtype == torch.bfloat16:
            o, ht = _ops.load().rwkv7_varlen(r, w, k, v, a, b, p.start, p.lens, p.max_len, initial_state)
            return (o, ht) if output_final_state else o
    except Exception as e:
        _check_args(r, w, k, v, a, b, initial_state, cu_seqlens)
        raise _ops.failed(e)
    n_seq = p.start.numel()
    if initial_state is not None and initial_state.shape[0] not in (1, n_seq):
        raise ValueError(f"initial_state must hold 1 or {n_seq} states, got {tuple(initial_state.shape)}")
    # one dense call per sequence (the float32 recurrence has no packed form)
    outs, states = [], []
    args = _token_args(r, w, k, v, a, b)
    for i in range(n_seq):
        s, e = int(p.cu[i]), int(p.cu[i + 1])
        hi = None if initial_state is None else initial_state[i:i + 1] if initial_state.shape[0] == n_seq else initial_state
        oi, si = generalized_delta_rule(*(x[:, s:e] for x in args), initial_state=hi)
        outs.append(oi)
        states.append(si)
    o, ht = torch.cat(outs, dim=1), torch.cat(states, dim=0)
    return (o, ht) if output_final_state else o


# ---------------------------------------------------------------------------------------------------------
# RWKV6 wkv on packed batches
# ---------------------------------------------------------------------------------------------------------
def _check_wkv6_args(r, k, v, w, u, cu_seqlens, init_state, state_map, head_size):
    """Raise what the interface documents for invalid arguments (the operator itself only says that they are)."""
    dev = _lib.require_cuda(r, k, v, w, u, init_state)
    if head_size != 64:
        raise ValueError("the packed wkv6 operator is built for head size 64")
    if r.dim() != 3 or r.shape[0] != 1 or r.shape[-1] % 64:
        raise ValueError(f"expected packed token tensors [1, total_len, H*64], got {tuple(r.shape)}")
    for name, x in (("k", k), ("v", v), ("w", w)):
        if x.shape != r.shape or x.dtype != r.dtype:
            raise ValueError(f"{name} must match r in shape and dtype")
    H, N = r.shape[2] // 64, 64
    if u.numel() != H * N:
        raise ValueError(f"u must have {H * N} elements")
    if isinstance(cu_seqlens, PackedSequences) and (cu_seqlens.total_len != r.shape[1] or cu_seqlens.start.device != dev):
        raise ValueError("the PackedSequences object was made for another token count or device")
    n_seq = cu_seqlens.start.numel() if isinstance(cu_seqlens, PackedSequences) else torch.as_tensor(cu_seqlens).numel() - 1
    if init_state is not None:
        if init_state.dim() not in (3, 4) or tuple(init_state.shape[-3:]) != (H, N, N):
            raise ValueError(f"init_state must be [n_state, {H}, {N}, {N}] or [{H}, {N}, {N}]")
        n_state = 1 if init_state.dim() == 3 else init_state.shape[0]
        if state_map is None and n_state not in (1, n_seq):
            raise ValueError("state_map cannot be inferred from init_state; pass it explicitly")
        if state_map is not None and torch.as_tensor(state_map).numel() != n_seq:
            raise ValueError("state_map must have one entry per sequence")
    elif state_map is not None:
        raise ValueError("state_map needs init_state")


def wkv6_varlen(r, k, v, w, u, cu_seqlens, init_state=None, state_map=None, head_size: int = 64):
    """The RWKV6 wkv operator over sequences packed end to end.

    The reference's operator takes dense ``[B, T, C]`` batches only (``rwkv_ops/rwkv6_kernel/
    ops_rwkv_kernel.py:10-21``); this is the same recurrence per sequence without a padded token ever loaded,
    computed or stored.  ``r, k, v, w``: ``[1, total_len, C]`` (or ``[total_len, C]``), ``C = H * 64``;
    ``u``: ``C`` elements; ``cu_seqlens``: ``n_seq + 1`` increasing integers from 0 to ``total_len`` (tensor,
    list or ``PackedSequences``); ``init_state``: ``[n_state, H, 64, 64]`` or ``[H, 64, 64]`` and ``state_map``
    ``[n_seq]`` as in the dense operator, with the sequence in the place of the batch row.  Returns
    ``(y, state)``: ``y`` shaped like ``r``, ``state`` ``[n_seq, H, 64, 64]`` in the operator's state dtype.
    Differentiable with respect to ``r, k, v, w, u`` and ``init_state``.
    """
    squeeze = r.dim() == 2
    if squeeze:
        r, k, v, w = (x[None] for x in (r, k, v, w))
    host_map = state_map
    try:
        if isinstance(cu_seqlens, PackedSequences) and r.dim() == 3 and cu_seqlens.total_len == r.shape[1] \
                and cu_seqlens.start.device == r.device and head_size == 64:
            p = cu_seqlens
        else:
            _check_wkv6_args(r, k, v, w, u, cu_seqlens, init_state, state_map, head_size)
            p = cu_seqlens if isinstance(cu_seqlens, PackedSequences) else _pack(cu_seqlens, r.shape[1], r.device)
        if state_map is not None:
            if isinstance(state_map, (list, tuple)):
                host_map = state_map = torch.tensor(state_map, dtype=torch.int32)
            if init_state is None:
                raise ValueError("state_map needs init_state")
            n_state = 1 if init_state.dim() == 3 else init_state.shape[0]
            if not state_map.is_cuda and not (bool((state_map >= 0).all()) and bool((state_map < n_state).all())):
                raise ValueError(f"state_map values must lie in [0, {n_state})")
            state_map = state_map.to(r.device, torch.int32)      # (any dtype that holds whole numbers)
        y, sT = _ops.load().wkv6_varlen(r, k, v, w, u, p.start, p.lens, p.max_len, init_state, state_map)
    except Exception as e:
        _check_wkv6_args(r, k, v, w, u, cu_seqlens, init_state, host_map, head_size)
        raise _ops.failed(e)
    return (y[0] if squeeze else y), sT
