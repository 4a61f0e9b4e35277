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


def _models():
    import ferrum_b200 as fb
    from ferrum_b200 import nn
    from ferrum_b200.models import wide_mlp

    dev = fb.Device.Cuda(0)
    return {"mlp": (wide_mlp(32, 64, 2, 16, device=dev), torch.randn(24, 32, device="cuda")),
            "encoder": (nn.TransformerEncoderLayer(64, 1, 128, device=dev), torch.randn(2, 130, 64, device="cuda")),
            "lstm": (nn.LSTM(8, 40, 2, device=dev), torch.randn(5, 3, 8, device="cuda"))}


def _grads(model, x, low, call):
    import ferrum_b200 as fb
    from ferrum_b200 import nn

    model.zero_grad()
    with fb.autocast(enabled=low):
        y = call(model, x)
        y2 = y.reshape(-1, y.shape[-1])
        t = torch.arange(y2.shape[0], device="cuda") % y2.shape[1]
        loss = nn.cross_entropy(y2, t) + nn.mse_loss(y, torch.zeros_like(y))
    loss.backward()
    return [p.grad.clone() for _, p in model.named_parameters()]


@pytest.mark.parametrize("name,low", [("mlp", False), ("mlp", True), ("encoder", False), ("encoder", True),
                                      ("lstm", False)])
def test_saved_tensor_hooks(name, low):
    """Hooks that move what the graph keeps to the host and back change no gradient and leave next to nothing on the GPU;
    non-reentrant checkpointing, which is built on them, gives the same gradients."""
    import ferrum_b200 as fb

    torch.manual_seed(5)
    model, x = _models()[name]
    want = _grads(model, x, low, lambda m, v: m(v))

    def check(got):
        # the encoder's column sums add in any order: its gradients repeat to a few roundings of the largest one
        top = max(t.abs().max().item() for t in want)
        for a, b in zip(got, want):
            assert torch.equal(a, b) if name != "encoder" else (a - b).abs().max() <= (2e-2 if low else 1e-5) * top

    to_host = lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda())
    with to_host():
        check(_grads(model, x, low, lambda m, v: m(v)))
    before = torch.cuda.memory_allocated()
    with to_host(), fb.autocast(enabled=low):
        y = model(x)
    # the result and, at most, a few blocks of the allocator's smallest size
    assert torch.cuda.memory_allocated() - before <= y.numel() * y.element_size() + 4 * 512
    del y

    def inner(v):  # the precision is the thread's: set inside, the recomputation runs in the engine's thread
        with fb.autocast(enabled=low):
            return model(v)

    check(_grads(model, x, low, lambda m, v: torch.utils.checkpoint.checkpoint(inner, v, use_reentrant=False)))
