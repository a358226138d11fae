"""Element by element, the decay gradient of tokens that decay slowly, or not at all, among faster ones."""
import pytest
import torch

import rwkv_ops_b200 as ro
from oracle import rwkv7_manual_backward
from rwkv_ops_b200.workloads import rwkv7_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("packed", [False, True])
def test_slow_and_masked_tokens_among_fast_ones(packed):
    """Half of the tokens of every channel at exp(w) in [1, 1.7], half at e^-11 .. e^-8, all inside the range of the chunked
    kernels; the first token of the second quarter of every chunk masked (w = -1e9: no decay, so no gradient)."""
    T, H = 200, 2
    d = rwkv7_inputs(1, T, H, dtype=torch.bfloat16, seed=31, with_grads=True)
    gen = torch.Generator().manual_seed(32)
    slow = torch.rand(d["w"].shape, generator=gen) < 0.5
    w = torch.where(slow, -11 + 3 * torch.rand(d["w"].shape, generator=gen), 0.55 * torch.rand(d["w"].shape, generator=gen))
    w[:, 16::64] = -1e9
    slow[:, 16::64] = False
    d["w"] = w.bfloat16()
    ref = rwkv7_manual_backward(*[d[n].double() for n in "rwkvab"], None, d["d_out"].double(), d["d_state"].double())[1]

    x = {n: d[n].cuda().requires_grad_(True) for n in "rwkvab"}
    if packed:      # 72 tokens of another sequence in front: the last chunk of both is stored row by row
        front = rwkv7_inputs(1, 72, H, dtype=torch.bfloat16, seed=33)
        y = {n: torch.cat([front[n].cuda(), x[n].detach()], 1).requires_grad_(True) for n in "rwkvab"}
        o, s = ro.generalized_delta_rule_varlen(*[y[n] for n in "rwkvab"], [0, 72, 72 + T])
        d_o = torch.cat([torch.zeros_like(front["r"]), d["d_out"]], 1).cuda()
        d_s = torch.cat([torch.zeros_like(d["d_state"]), d["d_state"]], 0).cuda()
        torch.autograd.backward([o, s], [d_o, d_s])
        dw = y["w"].grad[:, 72:].double().cpu()
    else:
        o, s = ro.generalized_delta_rule(*[x[n] for n in "rwkvab"])
        torch.autograd.backward([o, s], [d["d_out"].cuda(), d["d_state"].cuda()])
        dw = x["w"].grad.double().cpu()
    assert torch.equal(dw[:, 16::64], torch.zeros_like(dw[:, 16::64]))
    # dw = dg g: an error of dg (bfloat16 operands) is an absolute one, 0.4 % of the rms of dg; an error of g is
    # proportional to dg.  Entries with a dg of at least its rms: 2^-9 of rounding, 4 sigma of 0.4 %, and nothing from g.
    g = -torch.exp(d["w"].double())
    dg = ref[slow] / g[slow]
    big = dg.abs() >= dg.pow(2).mean().sqrt()
    err = ((dw[slow] - ref[slow]).abs() / ref[slow].abs())[big]
    assert float(err.max()) < 0.03, float(err.max())
    assert float((dw[slow] - ref[slow]).norm() / ref[slow].norm()) < 0.005
