"""What a backward pass keeps: results and inputs that a user may change in place, and tensors that saved-tensor hooks
see."""
import pytest
import torch
import torch.utils.checkpoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_logits_changed_after_cross_entropy(dtype):
    from ferrum_b200 import nn

    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(40, 304, device="cuda", generator=g).to(dtype).requires_grad_(True)
    t = torch.randint(0, 304, (40,), device="cuda", generator=g)
    grads = []
    for change in (False, True):
        x.grad = None
        logits = x * 1
        loss = nn.cross_entropy(logits, t)
        if change:
            logits.detach().zero_()
            logits.sigmoid_()
        loss.backward()
        grads.append(x.grad)
    assert torch.equal(*grads)


@pytest.mark.parametrize("kind", ["mse", "l1"])
def test_bf16_predictions_changed_after_the_loss(kind):
    from ferrum_b200 import nn

    x, t = (torch.randn(6, 5, device="cuda").bfloat16() for _ in range(2))
    x.requires_grad_(True)
    grads = []
    for change in (False, True):
        x.grad = None
        p = x * 1
        loss = getattr(nn, f"{kind}_loss")(p, t.clone())
        if change:
            p.mul_(2)
        loss.backward()
        grads.append(x.grad)
    assert torch.equal(*grads)


@pytest.mark.parametrize("kind", ["LSTM", "GRU"])
def test_sequence_output_changed_in_place(kind):
    import ferrum_b200 as fb
    from ferrum_b200 import nn

    torch.manual_seed(3)
    m = getattr(nn, kind)(8, 40, 2, device=fb.Device.Cuda(0))
    x, mask = torch.randn(5, 3, 8, device="cuda"), (torch.rand(5, 3, 40, device="cuda") > 0.5).float()
    grads = []
    for inplace in (False, True):
        m.zero_grad()
        y, last = m.forward_seq(x)
        y = y.mul_(mask) if inplace else y * mask
        (y.sum() + sum(t.sum() for t in (last if kind == "LSTM" else (last,)))).backward()
        grads.append([p.grad.clone() for _, p in m.named_parameters()])
    for a, b in zip(*grads):
        assert torch.equal(a, b)
