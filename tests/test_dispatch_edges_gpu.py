"""The kernels a call is dispatched to by its size and types, at the edges of their blocks: the scans for few and for
many sequences, the float32 recurrence over blocks of tokens, and wkv6 with few units or bfloat16 states."""
import pytest
import torch

import rwkv_ops_b200 as ro
from rwkv_ops_b200 import _lib
from oracle import generalized_delta_rule as oracle_gdr
from rwkv_ops_b200.workloads import rwkv7_inputs, wkv6_inputs, rel_l2

pytestmark = pytest.mark.gpu


def _train(d, grads, fn=ro.generalized_delta_rule):
    g = {n: d[n].clone().requires_grad_(True) for n in "rwkvab"}
    h0 = d["initial_state"].clone().requires_grad_(True)
    o, s = fn(*[g[n] for n in "rwkvab"], initial_state=h0)
    torch.autograd.backward([o, s], grads)
    return {"o": o.detach(), "s": s.detach(), "dh0": h0.grad, **{f"d{n}": g[n].grad for n in "rwkvab"}}


# one to six chunks: the chunk counts at which the accumulators and the operand buffers of the scans wrap around
@pytest.mark.parametrize("T", [8, 64, 65, 129, 200, 257, 384])
def test_scans_for_few_and_many_sequences(T):
    """Two units on their own (one CTA per SM) and among more units than there are SMs (two CTAs per SM)."""
    d = {n: t.cuda() for n, t in rwkv7_inputs(1, T, 2, dtype=torch.bfloat16, seed=70 + T, with_state=True, with_grads=True).items()}
    few = _train(d, [d["d_out"], d["d_state"]])
    ref = _train({n: t.float().cpu() for n, t in d.items()}, [d["d_out"].float().cpu(), d["d_state"].float().cpu()], oracle_gdr)
    for n in ref:
        assert rel_l2(few[n], ref[n]) < 2e-2, n
    B = torch.cuda.get_device_properties(0).multi_processor_count // 2 + 4
    big = {n: t.expand(B, *t.shape[1:]).contiguous() for n, t in d.items()}
    many = _train(big, [big["d_out"], big["d_state"]])
    for n in few:
        for row in (0, B - 1):
            assert rel_l2(many[n][row], few[n][0]) < 2e-3, n


@pytest.mark.parametrize("T", [1, 2, 7, 8, 9, 15, 16, 17, 33, 48])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float16, 2e-3)])
def test_token_blocks(T, dtype, tol):
    """Blocks of 8 tokens in the sweeps, items of 16 in the gradient kernel."""
    d = rwkv7_inputs(2, T, 3, dtype=dtype, seed=40 + T, with_state=True, with_grads=True)
    ref = _train({n: t.double() for n, t in d.items()}, [d["d_out"].double(), d["d_state"].double()], oracle_gdr)
    out = _train({n: t.cuda() for n, t in d.items()}, [d["d_out"].cuda(), d["d_state"].cuda()])
    for n in ref:
        assert rel_l2(out[n], ref[n]) < tol, n


@pytest.mark.parametrize("T", [1, 9, 64, 65, 200])
@pytest.mark.parametrize("many", [False, True])
def test_wkv6_states_in_the_token_dtype(T, many):
    """bfloat16 u, state table and final state, read and written as they are, against the call that converts them."""
    H = 2
    B = torch.cuda.get_device_properties(0).multi_processor_count // H + 4 if many else 2
    d = {n: t.cuda() for n, t in wkv6_inputs(B, T, H, dtype=torch.bfloat16, seed=20 + T, n_state=3).items()}
    s0, u = d["init_state"].bfloat16(), d["u"].bfloat16()
    smap = torch.arange(B, device="cuda", dtype=torch.int32) % 3
    op = ro.RWKV6_OP(64, T)
    with torch.no_grad():
        y, s = op(d["r"], d["k"], d["v"], d["w"], u, with_state=True, init_state=s0, state_map=smap)
        y32, s32 = op(d["r"], d["k"], d["v"], d["w"], u.float(), with_state=True, init_state=s0.float(), state_map=smap)
    assert y.dtype == s.dtype == torch.bfloat16
    assert torch.equal(y, y32) and torch.equal(s, s32.to(torch.bfloat16))


@pytest.mark.parametrize("T", [64 * 9, 64 * 17 - 5, 64 * 40 + 1])
def test_stages_of_the_scans_for_few_sequences_wrap_around(T):
    """Chunks enough to fill every stage of operand tiles several times over, against the recurrence; no wait runs out."""
    d = {n: t.cuda() for n, t in rwkv7_inputs(1, T, 2, dtype=torch.bfloat16, seed=90, with_state=True, with_grads=True).items()}
    lib = _lib.load()
    lib.rwkvb200_device_status(1)
    out = _train(d, [d["d_out"], d["d_state"]])
    assert lib.rwkvb200_device_status(1) == 0
    ref = _train({n: t.float() for n, t in d.items()}, [d["d_out"].float(), d["d_state"]])
    for n in ref:
        assert rel_l2(out[n], ref[n]) < 2e-2, n


def _recurrence(d, monkeypatch, grads):
    monkeypatch.setenv("RWKV_OPS_B200_RWKV7_ALGO", "recurrent")
    ref = _train(d, grads)
    monkeypatch.delenv("RWKV_OPS_B200_RWKV7_ALGO")
    return ref


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("T", [3, 7, 8, 15, 17, 33, 130])
def test_units_recomputed_inside_both_scans(T, many, monkeypatch):
    """Every third unit out of the range of the chunked kernels (all of them below 8 tokens), with one CTA per SM and with more
    units than SMs: those carry the bits of the recurrence, forward and backward, and the others stay the chunked kernels'."""
    H = 2
    B = torch.cuda.get_device_properties(0).multi_processor_count // H + 5 if many else 5
    d = {n: t.cuda() for n, t in rwkv7_inputs(B, T, H, dtype=torch.bfloat16, seed=50 + T, with_state=True, with_grads=True).items()}
    grads = [d["d_out"], d["d_state"]]
    inside = _train(d, grads)
    # 1.9 .. 2.9 per token leaves the range (60 per 32 tokens) only where half a chunk is that long
    fast = torch.zeros(B * H, dtype=torch.bool, device="cuda")
    fast[1::3] = T > 8
    w = torch.where(fast.view(B, 1, H, 1), (3.0 if T < 64 else 1.0) + 0.1 * d["w"].float(), d["w"].float()).bfloat16()
    if 8 <= T < 16:
        w = torch.where(fast.view(B, 1, H, 1), 3.0 + 0 * w, w)      # 15 tokens of e^3
    d["w"] = w
    out, ref = _train(d, grads), _recurrence(d, monkeypatch, grads)
    exact = torch.ones_like(fast) if T < 8 else fast
    for n in ref:
        a, b, c = (t.view(B, -1, H, 64, 64) if n in ("s", "dh0") else t for t in (out[n], ref[n], inside[n]))
        if n in ("s", "dh0"):
            a, b, c = (t.permute(0, 2, 1, 3, 4).reshape(B * H, -1) for t in (a, b, c))
        else:
            a, b, c = (t.permute(0, 2, 1, 3).reshape(B * H, -1) for t in (a, b, c))
        assert torch.equal(a[exact], b[exact]), n
        assert torch.equal(a[~exact], c[~exact]), n


def test_short_sequences_in_a_packed_batch_with_more_units_than_SMs(monkeypatch):
    """Sequences of 1 to 9 tokens between longer ones: those below 8 carry the bits of the recurrence over the sequence alone."""
    H, lens = 4, [1, 70, 2, 7, 8, 9, 130, 3] * 6
    assert len(lens) * H > torch.cuda.get_device_properties(0).multi_processor_count
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    d = rwkv7_inputs(1, cu[-1], H, dtype=torch.bfloat16, seed=77, device="cuda", with_grads=True)
    h0 = 0.1 * torch.randn(len(lens), H, 64, 64, device="cuda")
    d_s = 0.1 * torch.randn(len(lens), H, 64, 64, device="cuda")

    def run(fn, x, state, d_o, d_state):
        x = [t.clone().requires_grad_(True) for t in x]
        state = state.clone().requires_grad_(True)
        o, s = fn(*x, initial_state=state)
        return [o.detach(), s.detach(), *torch.autograd.grad([o, s], x + [state], [d_o, d_state])]

    tokens = [d[n] for n in "rwkvab"]
    out = run(lambda *x, **kw: ro.generalized_delta_rule_varlen(*x, cu, **kw), tokens, h0, d["d_out"], d_s)
    for i, n in enumerate(lens[:8]):
        at = slice(cu[i], cu[i] + n)
        monkeypatch.setenv("RWKV_OPS_B200_RWKV7_ALGO", "recurrent" if n < 8 else "auto")
        ref = run(ro.generalized_delta_rule, [t[:, at].contiguous() for t in tokens], h0[i:i + 1], d["d_out"][:, at].contiguous(), d_s[i:i + 1])
        monkeypatch.delenv("RWKV_OPS_B200_RWKV7_ALGO")
        for m, (a, b) in enumerate(zip(out, ref)):
            a = a[i:i + 1] if m in (1, 8) else a[:, at]
            if 1 < n < 8:
                assert torch.equal(a, b), (n, m)
            else:      # (one token alone is the decode step's kernel: other sums in float32, then perhaps another rounding)
                assert rel_l2(a, b) < 2e-3, (n, m)


@pytest.mark.parametrize("K", [64, 128])
@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 24, 33, 75])
def test_token_blocks_with_more_units_than_SMs(K, T):
    """Fewer preparing groups per CTA, down to one, and as many as there are blocks: the same bits as with few units."""
    d = rwkv7_inputs(1, T, 2, K, dtype=torch.float32, seed=40 + T, device="cuda", with_state=True, with_grads=True)
    few = _train(d, [d["d_out"], d["d_state"]])
    B = torch.cuda.get_device_properties(0).multi_processor_count // (K // 8) + 2
    big = {n: t.expand(B, *t.shape[1:]).contiguous() for n, t in d.items()}
    many = _train(big, [big["d_out"], big["d_state"]])
    for n in few:
        assert torch.equal(many[n], few[n].expand_as(many[n])), n


@pytest.mark.parametrize("K,dtype", [(64, torch.float32), (64, torch.float16), (128, torch.float32), (128, torch.bfloat16)])
@pytest.mark.parametrize("T", [16, 17, 32, 33, 70])
def test_states_kept_for_the_backward(T, K, dtype, monkeypatch):
    """The float32 recurrence's backward from the states its forward left (none up to 16 tokens), twice through the same graph,
    and from a second sweep: the same bits."""
    d = rwkv7_inputs(2, T, 3, K, dtype=dtype, seed=60 + T, device="cuda", with_state=True, with_grads=True)

    def grads():
        x = [d[n].clone().requires_grad_(True) for n in (*"rwkvab", "initial_state")]
        out = ro.generalized_delta_rule(*x[:6], initial_state=x[6])
        return [torch.autograd.grad(out, x, [d["d_out"], d["d_state"]], retain_graph=True) for _ in range(2)]

    kept = grads()
    monkeypatch.setenv("RWKV_OPS_B200_KEEP_LIMIT_MB", "0")
    again = grads()
    for a, b, c in zip(*kept, again[0]):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("K,dtype", [(64, torch.float32), (64, torch.float16), (128, torch.float32), (128, torch.bfloat16)])
@pytest.mark.parametrize("few", [False, True])
def test_blocks_prepared_apart(K, dtype, few):
    """The sweeps with and without their scratch (C ABI): the same bits, at the block counts from which the scratch is used, and
    just short of where a unit's blocks take several stretches of it."""
    lib, dev = _lib.load(), torch.device("cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    code = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}[dtype]
    H = 3 if few else 2 * sms // (K // 16) + 2
    for T in ((95, 96, 377, 384, 400) if few else (24, 25, 32, 33, 70)) + (() if few or K == 128 else (2500,)):
        d = rwkv7_inputs(1, T, H, K, dtype=dtype, seed=T, device="cuda", with_state=True)
        x = [d[n] for n in "rwkvab"]
        out = []
        for scratch in (True, False):
            o, s = torch.empty_like(x[0]), torch.empty(1, H, K, K, device=dev)
            n = lib.rwkvb200_rwkv7_fwd_workspace_bytes(1, T, H, K, code, _lib.ALGO_RECURRENT) if scratch else 0
            ws = torch.empty(n, dtype=torch.uint8, device=dev)
            _lib.check(lib.rwkvb200_rwkv7_fwd(*(_lib.ptr(t) for t in x), _lib.ptr(d["initial_state"]), 1, _lib.ptr(o), _lib.ptr(s),
                                              _lib.ptr(ws) if n else None, n, 1, T, H, K, code, 0, _lib.ALGO_RECURRENT,
                                              _lib.stream_ptr(dev)), "fwd")
            out.append((o, s))
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1]), T


def _sizes_prepared_apart(K, sms):
    """(units, tokens): block counts from which a sweep's blocks are prepared by a kernel of their own with fewer CTAs than SMs and
    with many; then stretches of blocks, and passes of units, where the scratch does not hold all of them."""
    return ([(3, T) for T in (95, 96, 377, 384, 400)] + [(2 * sms // (K // 16) + 2, T) for T in (24, 25, 32, 33, 70)]
            + [(400 if K == 64 else 200, 600), (3100 if K == 64 else 1200, 70)])


@pytest.mark.parametrize("K,dtype", [(64, torch.float32), (64, torch.float16), (128, torch.float32), (128, torch.bfloat16)])
def test_blocks_prepared_apart_forward_and_backward(K, dtype):
    """The sweeps of the forward and the backward, with and without states that the forward leaves, with and without their scratch
    (C ABI): the same bits, whatever part of it a call works with at a time."""
    lib, dev = _lib.load(), torch.device("cuda")
    code = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}[dtype]
    for H, T in _sizes_prepared_apart(K, torch.cuda.get_device_properties(0).multi_processor_count):
        d = rwkv7_inputs(1, T, H, K, dtype=dtype, seed=T, device="cuda", with_state=True, with_grads=True)
        x = [_lib.ptr(d[n]) for n in "rwkvab"]
        h0, d_o, d_ht = (_lib.ptr(d[n]) for n in ("initial_state", "d_out", "d_state"))
        size, end = (1, T, H, K, code, _lib.ALGO_RECURRENT), (1, T, H, K, code, 0, _lib.ALGO_RECURRENT, _lib.stream_ptr(dev))
        checkpoints = H * ((T + 7) // 8) * K * K * 4
        n_states = lib.rwkvb200_rwkv7_states_bytes(*size)
        assert n_states == _lib.rwkv7_states_bytes(1, T, H, K)

        def memory(n):
            return torch.empty(n, dtype=torch.uint8, device=dev)

        def run(scratch, kept):
            out = [torch.empty_like(d["r"]) for _ in range(7)] + [torch.empty(1, H, K, K, device=dev) for _ in range(2)]
            o, grads, ht, dh0 = _lib.ptr(out[0]), [_lib.ptr(t) for t in out[1:7]], _lib.ptr(out[7]), _lib.ptr(out[8])
            ws = memory(lib.rwkvb200_rwkv7_fwd_workspace_bytes(*size) if scratch else 0)
            fwd = (_lib.ptr(ws) if ws.numel() else None, ws.numel(), *end)
            if kept:
                states = memory(n_states)
                _lib.check(lib.rwkvb200_rwkv7_fwd_states(*x, h0, 1, o, ht, _lib.ptr(states), n_states, *fwd), "fwd_states")
                wb = memory(lib.rwkvb200_rwkv7_bwd_states_workspace_bytes(*size) if scratch else n_states)
                _lib.check(lib.rwkvb200_rwkv7_bwd_states(*x, h0, 1, d_o, d_ht, _lib.ptr(states), n_states, *grads, dh0, _lib.ptr(wb),
                                                         wb.numel(), *end), "bwd_states")
            else:
                _lib.check(lib.rwkvb200_rwkv7_fwd(*x, h0, 1, o, ht, *fwd), "fwd")
                wb = memory(lib.rwkvb200_rwkv7_bwd_workspace_bytes(*size) if scratch else (checkpoints + 255) // 256 * 256)
                _lib.check(lib.rwkvb200_rwkv7_bwd(*x, h0, 1, d_o, d_ht, *grads, dh0, _lib.ptr(wb), wb.numel(), *end), "bwd")
            return out

        ref = run(False, False)
        for scratch, kept in ((True, False), (False, True), (True, True)):
            for i, (got, want) in enumerate(zip(run(scratch, kept), ref)):
                assert torch.equal(got, want), (H, T, scratch, kept, i)


@pytest.mark.parametrize("H,T", [(2, 400), (80, 40)])
def test_blocks_prepared_apart_against_float64(H, T):
    """Training through the operator where the blocks are prepared apart: few units from 377 tokens on, many from 25 on."""
    d = rwkv7_inputs(1, T, H, dtype=torch.float32, seed=T, with_state=True, with_grads=True)
    ref = _train({n: t.double() for n, t in d.items()}, [d["d_out"].double(), d["d_state"].double()],
                 lambda *x, **kw: oracle_gdr(*x, **kw, compute_dtype=torch.float64))
    out = _train({n: t.cuda() for n, t in d.items()}, [d["d_out"].cuda(), d["d_state"].cuda()])
    for n in ref:
        assert rel_l2(out[n], ref[n]) < 1e-5, n


def test_scratch_that_cannot_be_had_is_done_without():
    """The float32 recurrence's scratch, and the states its forward leaves, are for speed: where the allocator has no room for
    them, the operator runs without and returns the same bits."""
    H, T, mb = 600, 512, 1 << 20
    d = rwkv7_inputs(1, T, H, seed=3, device="cuda", with_grads=True)
    x = [d[n].requires_grad_(True) for n in "rwkvab"]
    total = torch.cuda.get_device_properties(0).total_memory

    def room_for(more):      # what is in use, and `more` bytes
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + more) / total)

    tokens, states = x[0].numel() * 4, H * (T // 16 - 1) * 64 * 64 * 4
    try:
        o, s = ro.generalized_delta_rule(*x)
        grads = torch.autograd.grad([o, s], x, [d["d_out"], d["d_state"]], retain_graph=True)
        room_for(6 * tokens + states + 100 * mb)      # the backward's scratch are 256 MB more
        grads2 = torch.autograd.grad([o, s], x, [d["d_out"], d["d_state"]])
        assert all(torch.equal(a, b) for a, b in zip(grads, grads2))
        del grads2
        room_for(tokens + 100 * mb)                   # neither states nor scratch
        o2, s2 = ro.generalized_delta_rule(*x)
        assert torch.equal(o2, o) and torch.equal(s2, s)
        with torch.no_grad():
            del o2, s2
            room_for(tokens + 100 * mb)
            o2, s2 = ro.generalized_delta_rule(*x)
        assert torch.equal(o2, o) and torch.equal(s2, s)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


@pytest.mark.parametrize("lens,H", [([1500, 70, 64, 8, 200, 130, 9, 65, 300, 128], 20), ([8 + i % 70 for i in range(260)], 1),
                                    ([8 + 37 * i % 120 for i in range(700)], 3), ([70] * 255 + [2000], 2), ([1280, 70] * 20, 20)])
def test_scans_of_a_packed_batch_with_more_units_than_SMs(lens, H):
    """One sequence much longer than the others (its scans run one block to an SM, longest first), more sequences than are
    ranked by length, and two blocks to an SM, longest first; so many short sequences that a CTA's next chunk-head is a hundred of
    them on: as each sequence on its own."""
    assert len(lens) * H > torch.cuda.get_device_properties(0).multi_processor_count
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    d = rwkv7_inputs(1, cu[-1], H, dtype=torch.bfloat16, seed=31, device="cuda", with_grads=True)
    d_s = 0.1 * torch.randn(len(lens), H, 64, 64, device="cuda")

    def run(fn, x, d_o, d_state):
        x = [t.clone().requires_grad_(True) for t in x]
        o, s = fn(*x)
        return [s.detach(), o.detach(), *torch.autograd.grad([o, s], x, [d_o, d_state])]

    tokens = [d[n] for n in "rwkvab"]
    out = run(lambda *x: ro.generalized_delta_rule_varlen(*x, cu), tokens, d["d_out"], d_s)
    for i in {*range(min(len(lens), 10)), *range(10, len(lens), 97), len(lens) - 1}:
        at = slice(cu[i], cu[i + 1])
        ref = run(ro.generalized_delta_rule, [t[:, at].contiguous() for t in tokens], d["d_out"][:, at].contiguous(), d_s[i:i + 1])
        for m, (a, b) in enumerate(zip(out, ref)):
            assert rel_l2(a[i:i + 1] if m == 0 else a[:, at], b) < 2e-3, (i, m)


def _wkv6_train(d, call):
    x = [d[n].clone().requires_grad_(True) for n in "rkvwu"]
    y, s = call(*x)
    return [y.detach(), s.detach(), *torch.autograd.grad([y, s], x, [d["d_y"], d["d_state"].to(s.dtype)])]


# (sequences, tokens, heads): clusters of eight CTAs on their third lap and of two on their seventh; stretches on persistent CTAs.
# Tolerances of this file's other wkv6 tests; float16 rounds eight times finer than bfloat16.
@pytest.mark.parametrize("B,T,H", [(1, 1100, 2), (4, 777, 32), (5, 520, 64)])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2), (torch.float16, 2.5e-3)])
def test_wkv6_relays_and_stretches_against_the_recurrence(B, T, H, dtype, tol, monkeypatch):
    d = wkv6_inputs(B, T, H, dtype=dtype, seed=B + T, device="cuda", n_state=1, with_grads=True)
    op = ro.RWKV6_OP(64, T)

    def call(*x):
        return op(*x, with_state=True, init_state=d["init_state"], state_map=torch.zeros(B, dtype=torch.int32, device="cuda"))

    out = _wkv6_train(d, call)
    with torch.no_grad():
        y, s = call(*[d[n] for n in "rkvwu"])
    monkeypatch.setenv("RWKV_OPS_B200_WKV6_ALGO", "recurrent")
    ref = _wkv6_train(d, call)
    for i, (a, b) in enumerate(zip([*out, y, s], [*ref, ref[0], ref[1]])):
        assert rel_l2(a, b) < tol, i
    assert _lib.load().rwkvb200_device_status(1) == 0


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2), (torch.float16, 2.5e-3)])
def test_wkv6_relay_of_a_packed_batch(dtype, tol, monkeypatch):
    """Lengths on both sides of a chunk, a CTA's turn and a lap of the cluster; rows past a sequence's end belong to the next one."""
    lens, H = [512, 513, 63, 1031, 1, 64, 1088, 577], 2
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    d = wkv6_inputs(1, cu[-1], H, dtype=dtype, seed=9, device="cuda", n_state=1, with_grads=True)
    d["d_state"] = 0.1 * torch.randn(len(lens), H, 64, 64, device="cuda")
    out = _wkv6_train(d, lambda *x: ro.wkv6_varlen(*x, cu))
    monkeypatch.setenv("RWKV_OPS_B200_WKV6_ALGO", "recurrent")

    def one_by_one(r, k, v, w, u):
        ys = [ro.RWKV6_OP(64, n)(*(x[:, i:i + n] for x in (r, k, v, w)), u, with_state=True) for i, n in zip(cu, lens)]
        return torch.cat([y for y, _ in ys], 1), torch.cat([s for _, s in ys], 0)

    ref = _wkv6_train(d, one_by_one)
    for i, (a, b) in enumerate(zip(out, ref)):
        assert rel_l2(a, b) < tol, i
    assert _lib.load().rwkvb200_device_status(1) == 0


def _training_calls():
    """(name, inputs, call) of every path with more than one kernel: chunked, packed, fused, float32 by blocks, wkv6."""
    def rwkv7(name, dtype, B, T, H, fn=ro.generalized_delta_rule):
        d = rwkv7_inputs(B, T, H, dtype=dtype, seed=T, device="cuda", with_grads=True)
        return name, [d[n] for n in "rwkvab"], fn, [d["d_out"], d["d_state"]]

    yield rwkv7("chunked", torch.bfloat16, 2, 300, 8)
    yield rwkv7("chunked, many units", torch.bfloat16, 10, 130, 32)
    yield rwkv7("float32", torch.float32, 1, 400, 4)
    name, x, _, grads = rwkv7("packed", torch.bfloat16, 1, 700, 4)
    packed = ro.PackedSequences([0, 300, 310, 700])
    yield name, x, lambda *x: ro.generalized_delta_rule_varlen(*x, packed), [grads[0], grads[1].expand(3, -1, -1, -1).contiguous()]
    yield rwkv7("fused", torch.bfloat16, 2, 300, 8, ro.generalized_delta_rule_fused)
    for name, B, T, H in (("wkv6 relay", 1, 700, 4), ("wkv6 stretches", 5, 520, 64)):
        d = wkv6_inputs(B, T, H, dtype=torch.bfloat16, seed=T, device="cuda", with_grads=True)
        op = ro.RWKV6_OP(64, T)
        yield name, [d[n] for n in "rkvwu"], lambda *x, op=op: op(*x, with_state=True), [d["d_y"], d["d_state"].bfloat16()]


def _results(x, fn, grads):
    x = [t.detach().requires_grad_(True) for t in x]
    o, s = fn(*x)
    return [o, s, *torch.autograd.grad([o, s], x, grads)]


def _same(got, want, what):
    for i, (a, b) in enumerate(zip(got, want)):
        # (wkv6: the gradient of u, the last one, is summed by atomic additions)
        assert torch.equal(a, b) or (i == len(want) - 1 and "wkv6" in what and rel_l2(a, b) < 1e-2), (what, i)


def test_training_replays_from_a_cuda_graph():
    """Calls of several kernels, whose launches overlap, captured and replayed on other inputs."""
    for name, x, fn, grads in _training_calls():
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _results(x, fn, grads)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = _results(x, fn, grads)
        for _ in range(2):
            for t in x:
                t.copy_(t.flip(1).contiguous() if t.dim() > 2 else t.flip(0))
            graph.replay()
            _same(out, _results(x, fn, grads), name)
    assert _lib.load().rwkvb200_device_status(1) == 0


def test_training_on_two_streams_at_once():
    """Two calls of every pair of paths in flight at the same time: their kernels share SMs, and each keeps its own workspace."""
    calls = list(_training_calls())
    want = [_results(*call[1:]) for call in calls]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for i in range(len(calls)):
        for j in range(i, len(calls)):
            torch.cuda.synchronize()
            got = []
            for stream, c in zip(streams, (i, j)):
                with torch.cuda.stream(stream):
                    got.append([_results(*calls[c][1:]) for _ in range(3)])
            torch.cuda.synchronize()
            for c, results in zip((i, j), got):
                for r in results:
                    _same(r, want[c], calls[c][0])
    assert _lib.load().rwkvb200_device_status(1) == 0
