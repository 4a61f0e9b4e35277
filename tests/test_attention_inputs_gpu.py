"""Projections that share one bf16 copy of their input: the bits of three copies, with hooks, distinct inputs and an input
that needs a gradient on the general path."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("how", ["same", "distinct", "hook", "grad"])
def test_shared_input(train, how):
    import ferrum_b200 as fb
    import ferrum_b200.nn as nn

    torch.manual_seed(0)
    m = nn.MultiHeadAttention(128, 2, device=fb.Device.Cuda(0))
    x = torch.randn(2, 65, 128, device="cuda")
    args = [x, x, x] if how != "distinct" else [x, x.clone(), x.clone()]
    seen = []
    hook = m.k_proj.register_forward_pre_hook(lambda mod, a: seen.append(a[0].dtype)) if how == "hook" else None
    if how == "grad":
        x.requires_grad_(True)

    def run(a):
        with torch.set_grad_enabled(train), fb.autocast():
            y = m.forward_attn(*a)
        grads = []
        if train:
            for p in m.torch_parameters():
                p.grad = None
            y.float().square().sum().backward()
            grads = [p.grad.clone() for p in m.torch_parameters()]
        return [y.detach()] + grads

    got = run(args)
    if hook is not None:
        assert seen == [torch.float32]
        hook.remove()
    want = run([x.detach().clone() for _ in range(3)])
    assert torch.equal(got[0], want[0])
    # sums by atomics may differ in order; the key bias' gradient is zero in exact arithmetic, all rounding
    scale = max((float(b.norm()) for b in want[1:]), default=0.0)
    for a, b in zip(got[1:], want[1:]):
        assert (a - b).norm() <= 1e-5 * b.norm() + 1e-6 * scale
    if how == "grad" and train:
        assert x.grad is not None and x.grad.dtype == torch.float32
