"""The native ops have no forward-mode derivative: a dual input is refused, in either grad mode, instead of losing its
tangent."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

pytestmark = pytest.mark.gpu


def _calls(d):
    from ferrum_b200.ops import functional as F

    w, b, one = (torch.randn(*s, device="cuda") for s in ((6, 8), (6,), (8,)))
    t = torch.zeros(4, dtype=torch.int64, device="cuda")
    q = torch.randn(1, 1, 8, 4, device="cuda")
    return {
        "linear": lambda: F.linear(d, w, b),
        "linear_act_layernorm": lambda: F.linear_act_layernorm(d, w, b, b, b),
        "layer_norm": lambda: F.layer_norm(d, one, one),
        "unary": lambda: F.unary(d, "exp"),
        "add": lambda: F.binary(d, d, "add"),
        "softmax": lambda: F.softmax(d),
        "cross_entropy": lambda: F.cross_entropy_logits(d, t),
        "nll": lambda: F.nll_index(d, t),
        "mse": lambda: F.elementwise_loss(d, torch.zeros_like(w[:4, :1]).expand(4, 8), "mse"),
        "mse_target": lambda: F.elementwise_loss(torch.zeros(4, 8, device="cuda"), d, "mse"),
        "bmm": lambda: F.bmm_scaled(d.reshape(1, 1, 4, 8), q),
        "embedding": lambda: F.embedding(d, t),
        "rnn": lambda: F.rnn_sequence(4, d.reshape(4, 1, 8), torch.randn(8, 2, device="cuda"), None),
        "add_layer_norm": lambda: F.add_layer_norm(d, torch.zeros_like(w[:4]), one, one),
        "add_layer_norm_branch": lambda: F.add_layer_norm(torch.zeros_like(w[:4]), d, one, one),
        "conv2d": lambda: F.conv2d_igemm(d.reshape(1, 1, 4, 8), torch.randn(2, 1, 3, 3, device="cuda"), None),
    }


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("low", [True, False])
def test_attention_refuses_dual_inputs(grad, low):
    import ferrum_b200 as fb
    from ferrum_b200 import nn

    m = nn.MultiHeadAttention(128, 2, device=fb.Device.Cuda(0))
    x = torch.randn(1, 5, 128, device="cuda")
    with fwd.dual_level(), torch.set_grad_enabled(grad), fb.autocast(enabled=low):
        d = fwd.make_dual(x, torch.ones_like(x))
        for args in ((d, d, d), (d, x, x), (x, d, x), (x, x, d)):
            with pytest.raises(NotImplementedError):
                m.forward_attn(*args)
                pytest.fail("a tangent was lost")
        m.forward_attn(x, x, x)  # no tangent: nothing to refuse


@pytest.mark.parametrize("grad", [True, False])
def test_dual_inputs_are_refused(grad):
    with fwd.dual_level(), torch.set_grad_enabled(grad):
        d = fwd.make_dual(torch.randn(4, 8, device="cuda"), torch.ones(4, 8, device="cuda"))
        for name, call in _calls(d).items():
            with pytest.raises(NotImplementedError):
                call()
                pytest.fail(name)
