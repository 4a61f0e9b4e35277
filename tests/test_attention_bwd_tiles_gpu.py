"""Attention backward around its tiles (128 rows of the resident side, 64 of the walked one), against autograd in fp64.

Bound: P, dS and the results are rounded to bf16 (2^-9 each) and the forward output that enters the row sums, too: 2 % of
the norm covers the four roundings and their cancellation in dS."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Skv", [(1, 1), (63, 64), (64, 65), (65, 127), (128, 128), (129, 192), (200, 257), (320, 385), (449, 577)])
def test_gradients(Sq, Skv, D, causal):
    from ferrum_b200.ops import functional as F
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(Sq * 1000 + Skv + D)
    rand = lambda s: torch.randn(2, s, 3, D, device="cuda", generator=g).bfloat16()
    q, k, v = rand(Sq), rand(Skv), rand(Skv)
    gy = torch.randn(2, 3, Sq, D, device="cuda", generator=g).bfloat16()
    low = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = F.attention_blockwise(*(t.transpose(1, 2) for t in low), D ** -0.5, causal=causal)
    out.backward(gy)
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    qd, kd, vd = (t.transpose(1, 2) for t in ref)
    s = qd @ kd.transpose(-1, -2) * D ** -0.5
    if causal:
        i, j = torch.arange(Sq, device="cuda")[:, None], torch.arange(Skv, device="cuda")[None]
        s = s.masked_fill(j > i + (Skv - Sq), float("-inf"))
    want = torch.softmax(s, -1) @ vd
    want.backward(gy.double())
    check_status()
    assert (out.double() - want).norm() <= 0.01 * want.norm()
    scale = sum(t.grad.norm() for t in ref)  # with one key the gradients of q and k are zero
    for a, c in zip(low, ref):
        assert (a.grad.double() - c.grad).norm() <= 0.02 * c.grad.norm() + 1e-3 * scale
