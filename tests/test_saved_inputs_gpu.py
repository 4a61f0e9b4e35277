"""Labels, targets and indices changed between the forward and the backward pass are an error, never another gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["cross_entropy", "nll", "mse", "embedding"])
def test_changed_before_backward(kind):
    import ferrum_b200 as fb
    from ferrum_b200 import nn

    x = torch.randn(6, 5, device="cuda", requires_grad=True)
    t = torch.randint(0, 5, (6,), device="cuda")
    if kind == "cross_entropy":
        loss = nn.cross_entropy(x, t)
    elif kind == "nll":
        loss = nn.nll_loss(torch.log_softmax(x, -1), t)
    elif kind == "mse":
        t = torch.randn(6, 5, device="cuda")
        loss = nn.mse_loss(x, t)
    else:
        loss = nn.Embedding(5, 8, device=fb.Device.Cuda(0))(t).sum()
    t.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        loss.backward()
