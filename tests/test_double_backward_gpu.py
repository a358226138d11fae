"""Second derivatives are not built: asking for one raises; a first derivative with ``create_graph`` is what it is without."""
import pytest
import torch

import rwkv_ops_b200 as ro
from rwkv_ops_b200.workloads import rel_l2, rwkv7_inputs, wkv6_inputs

pytestmark = pytest.mark.gpu


def _rwkv7(dtype):
    return [t for n, t in rwkv7_inputs(2, 70, 2, dtype=dtype, seed=7, device="cuda").items()]


def _wkv6(B):
    d = wkv6_inputs(B, 70, 2, dtype=torch.float32, seed=8, device="cuda")
    return [d[n] for n in ("r", "k", "v", "w", "u")]


CALLS = {
    "rwkv7 bf16": (lambda: _rwkv7(torch.bfloat16), ro.generalized_delta_rule),
    "rwkv7 f32": (lambda: _rwkv7(torch.float32), ro.generalized_delta_rule),
    "rwkv7 packed": (lambda: [t[:1].contiguous() for t in _rwkv7(torch.bfloat16)],
                     lambda *x: ro.generalized_delta_rule_varlen(*x, [0, 30, 70])),
    "rwkv7 fused": (lambda: _rwkv7(torch.bfloat16), ro.generalized_delta_rule_fused),
    "wkv6": (lambda: _wkv6(2), lambda *x: ro.RWKV6_OP(64, 70)(*x, with_state=True)),
    "wkv6 packed": (lambda: _wkv6(1), lambda *x: ro.wkv6_varlen(*x, [0, 30, 70])),
}


@pytest.mark.parametrize("name", list(CALLS))
def test_second_derivative_raises(name):
    make, op = CALLS[name]
    x = [t.requires_grad_(True) for t in make()]

    def loss():
        o, s = op(*x)
        return o.float().square().sum() + s.float().sum()

    plain = torch.autograd.grad(loss(), x)
    grads = torch.autograd.grad(loss(), x, create_graph=True)
    for a, b in zip(plain, grads):
        assert b.requires_grad and rel_l2(b, a) < 1e-6      # (du is summed in no fixed order)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(sum(g.float().square().sum() for g in grads), x)
