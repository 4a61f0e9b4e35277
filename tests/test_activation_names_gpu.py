"""Activations of the fused layers: a name that no kernel evaluates is never the identity."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu


def _precision(low):
    import ferrum_b200 as fb

    return fb.autocast() if low else contextlib.nullcontext()


@pytest.mark.parametrize("low", [False, True])
@pytest.mark.parametrize("act", ["leaky_relu", "elu", "abs", "exp"])
def test_linear(act, low):
    from ferrum_b200.ops import functional as F

    x, w = torch.randn(16, 32, device="cuda"), torch.randn(24, 32, device="cuda")
    with _precision(low):
        with pytest.raises(KeyError):
            F.linear(x, w, None, act)
        y = F.linear(x, w.requires_grad_(True), None, act)  # recorded: a node of its own
        assert torch.equal(y, F.unary(F.linear(x, w, None), act))


@pytest.mark.parametrize("low", [False, True])
@pytest.mark.parametrize("K", [32, 33])
@pytest.mark.parametrize("act", [None, "gelu", "relu", "silu", "tanh", "sigmoid", "leaky_relu", "elu"])
def test_linear_act_layernorm(act, K, low):
    """Against fp64 torch; the bound is a few roundings of the result's type for values of order one."""
    from ferrum_b200.ops import functional as F

    g = torch.Generator(device="cuda").manual_seed(K)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).requires_grad_(True)
    x, w, b, gamma, beta = rand(64, K), rand(40, K), rand(40), rand(40), rand(40)
    up = torch.randn(64, 40, device="cuda", generator=g)
    with _precision(low):
        if low and K % 8 == 0 and act in ("leaky_relu", "elu"):  # the epilogue has no such activation
            with pytest.raises(KeyError):
                F.linear_act_layernorm(x, w, b, gamma, beta, act=act)
            return
        y = F.linear_act_layernorm(x, w, b, gamma, beta, act=act)
        y.backward(up.to(y.dtype))
    leaves = [t.detach().double().requires_grad_(True) for t in (x, w, b, gamma, beta)]
    z = torch.nn.functional.linear(*leaves[:3])
    z = z if act is None else {"gelu": lambda t: torch.nn.functional.gelu(t, approximate="tanh"),
                               # a name carries no parameter: alpha = 0 in both
                               "leaky_relu": lambda t: torch.nn.functional.leaky_relu(t, 0.0),
                               "elu": lambda t: torch.nn.functional.elu(t, 0.0)}.get(
        act, getattr(torch.nn.functional, act))(z)
    r = torch.nn.functional.layer_norm(z, (40,), leaves[3], leaves[4])
    r.backward(up.double())
    bound = 3e-2 if low else 2e-5
    for got, want in [(y, r)] + [(t.grad, s.grad) for t, s in zip((x, w, b, gamma, beta), leaves)]:
        assert (got.double() - want).norm() <= bound * want.norm() + 1e-5


@pytest.mark.parametrize("act", ["gelu", "silu", "relu"])
def test_bias_alone_trained(act):
    """The derivative of a GELU is no function of its output, whichever of the operands is trained."""
    from ferrum_b200.ops import functional as F

    x, w, b = (torch.randn(*s, device="cuda") for s in ((16, 32), (24, 32), (24,)))
    b.requires_grad_(True)
    F.linear(x, w, b, act).sum().backward()
    d = b.detach().double().requires_grad_(True)
    z = torch.nn.functional.linear(x.double(), w.double(), d)
    (torch.nn.functional.gelu(z, approximate="tanh") if act == "gelu" else getattr(torch.nn.functional, act)(z)).sum().backward()
    assert (b.grad.double() - d.grad).norm() <= 1e-5 * d.grad.norm()
