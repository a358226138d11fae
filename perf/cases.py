"""The operator calls whose speed is tracked: what a program that trains, prefills or decodes with RWKV7 / RWKV6
layers asks of this package, through the public entry points.

Every case is a plain dict; ``kind`` names the call:

==================  ==================================================================================
``step``            one decode step on a resident state (``Rwkv7DecodeState.step``)
``step_op``         one decode step through the operator (``T == 1``, the state fed back by the caller)
``prefill``         RWKV7 forward without gradients, final state returned
``train``           RWKV7 forward + backward, gradients of every token tensor (and of the initial state)
``train_packed``    the same over sequences packed end to end
``train_fused``     the same with the producers of w, a, b inside the operator
``wkv6_forward``    RWKV6 wkv forward without gradients, from a state table, final state returned
``wkv6_train``      RWKV6 wkv forward + backward, gradients of r, k, v, w, u and of the state table
==================  ==================================================================================

Values follow the distributions of ``rwkv_ops_b200.workloads``.
"""
import math
import random

import torch

from rwkv_ops_b200 import (RWKV6_OP, PackedSequences, Rwkv7DecodeState, generalized_delta_rule,
                           generalized_delta_rule_fused, generalized_delta_rule_varlen)
from rwkv_ops_b200.workloads import apply_w_padding, rwkv7_inputs, rwkv7_pad_lengths, wkv6_inputs

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32, "f16": torch.float16}
BYTES = {"bf16": 2, "f32": 4, "f16": 2}
TOKENS = ("r", "w", "k", "v", "a", "b")
PRE_TOKENS = ("r", "w_pre", "k", "v", "kk_pre", "a_pre")


def listed():
    return [
        # interactive generation: one sequence, one token of one layer; the call itself is all there is
        dict(name="decode, one sequence", kind="step", B=1, H=32, dtype="bf16", state="f32"),
        # a decode server's full batch, the state going in and out of the operator (benchmark configuration 3)
        dict(name="decode, batch of 256", kind="step_op", B=256, H=64, dtype="bf16"),
        # the same server at an odd moment, keeping its states in bfloat16 to hold more sequences
        dict(name="decode, bf16 state", kind="step", B=97, H=40, dtype="bf16", state="bf16"),
        # one user's prompt, of whatever length it has
        dict(name="prefill, one prompt", kind="prefill", B=1, T=1000, H=32, dtype="bf16", with_state=False),
        # a small model's micro-batch (fine-tuning on short texts)
        dict(name="train, small", kind="train", B=2, T=371, H=12, dtype="bf16", head=64, with_state=False, padded=False),
        # pre-training at 2048 channels (benchmark configuration 1)
        dict(name="train, 2048 channels", kind="train", B=8, T=4096, H=32, dtype="bf16", head=64, with_state=False,
             padded=False),
        # 4096 channels, long padded sequences that continue from a state (benchmark configuration 2)
        dict(name="train, 4096 channels", kind="train", B=16, T=8192, H=64, dtype="bf16", head=64, with_state=True,
             padded=True),
        # float32 tokens, for those who need float32-exact gradients
        dict(name="train, float32", kind="train", B=2, T=1024, H=16, dtype="f32", head=64, with_state=True, padded=False),
        # documents of very different lengths packed into one batch
        dict(name="train, packed", kind="train_packed", n_seq=8, max_len=4096, H=32),
        # a time-mix block that hands its pre-activations to the operator
        dict(name="train, fused producers", kind="train_fused", B=4, T=2000, H=32),
        # RWKV6 prefill of a few prompts, each from a state of a shared table
        dict(name="wkv6 forward", kind="wkv6_forward", B=4, T=777, H=32, dtype="bf16", n_state=4),
        # RWKV6 training in float32 (benchmark configuration 4)
        dict(name="wkv6 train, float32", kind="wkv6_train", B=16, T=4096, H=32, dtype="f32", n_state=4),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng: random.Random):
    kind = rng.choice(("step", "step_op", "prefill", "train", "train", "train", "train_packed", "train_fused",
                       "wkv6_forward", "wkv6_train", "wkv6_train"))
    H = rng.randint(8, 64)
    if kind == "step":
        return dict(kind=kind, B=_log_int(rng, 1, 256), H=H, dtype=rng.choice(("bf16", "bf16", "f16", "f32")),
                    state=rng.choice(("f32", "bf16")))
    if kind == "step_op":
        return dict(kind=kind, B=_log_int(rng, 1, 256), H=H, dtype=rng.choice(("bf16", "bf16", "f32")))
    B, T = _log_int(rng, 1, 16), _log_int(rng, 2, 8192)
    if kind == "prefill":
        return dict(kind=kind, B=B, T=T, H=H, dtype="bf16", with_state=rng.random() < 0.5)
    if kind == "train":
        dtype = rng.choice(("bf16", "bf16", "bf16", "f32", "f16"))
        head = 64
        if dtype != "bf16":      # token by token in float32: fewer and shorter sequences
            head = rng.choice((64, 64, 128))
            B, H, T = min(B, 4), min(H, 32), max(2, min(T, 1024) * 64 // head)
        return dict(kind=kind, B=B, T=T, H=H, dtype=dtype, head=head, with_state=rng.random() < 0.5,
                    padded=rng.random() < 0.3 and T >= 64)
    if kind == "train_packed":
        return dict(kind=kind, n_seq=_log_int(rng, 2, 24), max_len=_log_int(rng, 32, 6000), H=min(H, 48))
    if kind == "train_fused":
        return dict(kind=kind, B=B, T=T, H=H)
    dtype = rng.choice(("f32", "bf16"))
    if kind == "wkv6_forward":
        return dict(kind=kind, B=B, T=_log_int(rng, 1, 8192), H=H, dtype=dtype, n_state=rng.choice((1, 3, 4)))
    T = min(T, max(2, (16 * 4096 * 32) // (B * H)))
    return dict(kind=kind, B=B, T=T, H=H, dtype=dtype, n_state=rng.choice((1, 3, 4)))


def _lengths(case):
    """Sequence lengths of a packed batch: uniform in [max_len / 16, max_len], one of them max_len."""
    rng = random.Random("%d sequences of %d" % (case["n_seq"], case["max_len"]))
    lens = [rng.randint(max(1, case["max_len"] // 16), case["max_len"]) for _ in range(case["n_seq"])]
    lens[rng.randrange(len(lens))] = case["max_len"]
    return lens


def _offsets(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu


def prepare(case, seed):
    kind, H = case["kind"], case["H"]
    st = {"kind": kind}
    if kind in ("step", "step_op"):
        d = rwkv7_inputs(case["B"], 1, H, dtype=DTYPES[case["dtype"]], seed=seed, device="cuda", with_state=True)
        st["tokens"] = [d[n] for n in TOKENS]
        if kind == "step":
            st["decoder"] = Rwkv7DecodeState(case["B"], H, state_dtype=DTYPES[case["state"]],
                                             initial_state=d["initial_state"])
        else:
            st["state"] = d["initial_state"]
    elif kind in ("prefill", "train"):
        d = rwkv7_inputs(case["B"], case["T"], H, case.get("head", 64), dtype=DTYPES[case["dtype"]], seed=seed,
                         device="cuda", with_state=case["with_state"], with_grads=kind == "train")
        if case.get("padded"):
            d["w"] = apply_w_padding(d["w"], rwkv7_pad_lengths(case["B"], case["T"]))
        st["tokens"] = [d[n] for n in TOKENS]
        st["initial_state"] = d.get("initial_state")
        st["d_out"], st["d_state"] = d.get("d_out"), d.get("d_state")
    elif kind == "train_packed":
        lens = _lengths(case)
        d = rwkv7_inputs(1, sum(lens), H, dtype=torch.bfloat16, seed=seed, device="cuda", with_grads=True)
        st["tokens"] = [d[n] for n in TOKENS]
        st["sequences"] = PackedSequences(_offsets(lens), "cuda")      # made once for all the layers of a step
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        st["d_out"] = d["d_out"]
        st["d_state"] = 0.1 * torch.randn(len(lens), H, 64, 64, generator=g, device="cuda")
    elif kind == "train_fused":
        g = torch.Generator(device="cuda").manual_seed(seed)

        def normal(*shape):
            return torch.randn(*shape, generator=g, device="cuda")

        st["tokens"] = [normal(case["B"], case["T"], H, 64).bfloat16() for _ in PRE_TOKENS]
        st["d_out"] = normal(case["B"], case["T"], H, 64).bfloat16()
        st["d_state"] = 0.1 * normal(case["B"], H, 64, 64)
    else:
        d = wkv6_inputs(case["B"], case["T"], H, dtype=DTYPES[case["dtype"]], seed=seed, device="cuda",
                        n_state=case["n_state"], with_grads=kind == "wkv6_train")
        st["tokens"] = [d[n] for n in ("r", "k", "v", "w", "u")]
        st["initial_state"], st["state_map"] = d["init_state"], d["state_map"]
        st["d_out"], st["d_state"] = d.get("d_y"), d.get("d_state")
        st["op"] = RWKV6_OP(64, case["T"])
    if kind in ("train", "train_packed", "train_fused", "wkv6_train"):
        st["leaves"] = list(st["tokens"])
        if st.get("initial_state") is not None:
            st["leaves"].append(st["initial_state"])
        for t in st["leaves"]:
            t.requires_grad_(True)
    return st


def run(st):
    kind = st["kind"]
    if kind == "step":
        return {"o": st["decoder"].step(*st["tokens"]), "state": st["decoder"].state}
    if kind == "step_op":
        with torch.no_grad():
            o, st["state"] = generalized_delta_rule(*st["tokens"], initial_state=st["state"])
        return {"o": o, "state": st["state"]}
    if kind == "prefill":
        with torch.no_grad():
            o, s = generalized_delta_rule(*st["tokens"], initial_state=st["initial_state"])
        return {"o": o, "state": s}
    if kind == "wkv6_forward":
        with torch.no_grad():
            y, s = st["op"](*st["tokens"], with_state=True, init_state=st["initial_state"], state_map=st["state_map"])
        return {"o": y, "state": s}
    if kind == "train":
        o, s = generalized_delta_rule(*st["tokens"], initial_state=st["initial_state"])
    elif kind == "train_packed":
        o, s = generalized_delta_rule_varlen(*st["tokens"], st["sequences"])
    elif kind == "train_fused":
        o, s = generalized_delta_rule_fused(*st["tokens"])
    else:
        o, s = st["op"](*st["tokens"], with_state=True, init_state=st["initial_state"], state_map=st["state_map"])
    grads = torch.autograd.grad([o, s], st["leaves"], [st["d_out"], st["d_state"]])
    return {"o": o.detach(), "state": s.detach(), "grads": list(grads)}


def work(case):
    """Bytes: every input and every output once.  Operations: those of the token-by-token recurrence (a chunked
    evaluation does more): per token and head of N x N state, RWKV7 forward 9 N^2 (S a, the update, S r) and
    backward 20 N^2, RWKV6 forward 5 N^2 and backward 10 N^2."""
    kind, H = case["kind"], case["H"]
    N = case.get("head", 64)
    e = BYTES[case.get("dtype", "bf16")]
    if kind in ("step", "step_op"):
        units = case["B"] * H
        se = BYTES[case.get("state", "f32")]
        return {"bytes": units * (2 * N * N * se + 7 * N * e), "flops": units * 9 * N * N}
    if kind == "train_packed":
        rows, n_seq = sum(_lengths(case)) * H, case["n_seq"]
    else:
        rows, n_seq = case["B"] * case["T"] * H, case["B"]
    state = n_seq * H * N * N
    if kind == "prefill":
        return {"bytes": rows * N * e * 7 + state * 4 * (2 if case["with_state"] else 1), "flops": rows * 9 * N * N}
    if kind == "wkv6_forward":
        return {"bytes": rows * N * e * 5 + (case["n_state"] * H * N * N + state) * e, "flops": rows * 5 * N * N}
    if kind == "wkv6_train":
        # in r k v w dy, out y dr dk dv dw; final state and its gradient; the table and its gradient
        return {"bytes": rows * N * e * 10 + (2 * state + 2 * case["n_state"] * H * N * N) * e,
                "flops": rows * 15 * N * N}
    # in r w k v a b do, out o dr dw dk dv da db; final state and its gradient (the initial one and its gradient)
    return {"bytes": rows * N * e * 14 + state * 4 * (4 if case.get("with_state") else 2), "flops": rows * 29 * N * N}


def tolerance(case):
    kind = case["kind"]
    if kind in ("step", "step_op"):
        half = case["dtype"] != "f32" or case.get("state") == "bf16"
        return {"rel": 5e-3} if half else {"rel": 1e-5}
    if kind == "train" and case["dtype"] == "f16":
        return {"rel": 2e-3}
    if kind in ("wkv6_forward", "wkv6_train") and case["dtype"] == "f32":
        return {"rel": 1e-4}      # operands of 16 significant bits, decay gradients that are differences of sums
    if case.get("dtype", "bf16") == "f32":
        return {"rel": 1e-5}
    return {"rel": 1e-2}
