"""Convolutions as implicit GEMMs with what is fused around them: a ReLU, an added tensor, strides larger than the kernel,
channel counts that are no multiple of 8.  Against an fp64 convolution of the bf16-rounded operands.

Bound: products of bf16 numbers are exact in fp32 and at most a few thousand are added (1e-5 of the norm); gradients pass
through one more bf16 rounding of the incoming gradient, which the reference makes, too."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _r16(t):
    return t.bfloat16().double()


def _close(got, want):
    assert (got.double() - want).norm() <= 2e-5 * want.norm() + 1e-6


@pytest.mark.parametrize("fused", [None, "relu", "add"])
@pytest.mark.parametrize("B,C,O,H,W,k,stride,pad,dil", [
    (2, 8, 16, 9, 11, (3, 3), (1, 1), (1, 1), (1, 1)), (1, 3, 5, 17, 19, (3, 3), (2, 2), (1, 1), (1, 1)),
    (3, 64, 130, 28, 28, (1, 1), (2, 2), (0, 0), (1, 1)), (2, 65, 64, 14, 13, (2, 1), (3, 2), (1, 0), (1, 1)),
    (1, 128, 72, 7, 70, (3, 3), (1, 1), (2, 2), (2, 2)), (2, 12, 24, 33, 31, (5, 3), (2, 3), (2, 1), (1, 1)),
    (1, 24, 8, 32, 32, (4, 4), (4, 4), (0, 0), (1, 1)), (1, 1, 1, 1, 1, (1, 1), (1, 1), (0, 0), (1, 1))])
def test_forward_and_backward(B, C, O, H, W, k, stride, pad, dil, fused):
    import ferrum_b200 as fb
    from ferrum_b200.ops import functional as F
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(C + O + H)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, b = rand(B, C, H, W).requires_grad_(True), (rand(O, C, *k) * 0.1).requires_grad_(True), rand(O).requires_grad_(True)
    xd, wd, bd = _r16(x.detach()).requires_grad_(True), _r16(w.detach()).requires_grad_(True), b.detach().double().requires_grad_(True)
    zd = torch.nn.functional.conv2d(xd, wd, bd, stride, pad, dil)
    add = rand(*zd.shape).requires_grad_(True) if fused == "add" else None
    with fb.autocast():
        assert F.conv_igemm_ok(x, stride, dil, pad, k, 1)
        y = F.conv2d_igemm(x, w, b, pad, dil, stride, add, "relu" if fused == "relu" else None)
    gy = rand(*zd.shape)
    if fused == "relu":
        kept = y.detach() > 0  # next to zero either side is right
        yd, gd = zd * kept, gy * kept
        assert zd.detach()[kept != (zd > 0)].abs().sum() < 1e-3
    else:
        yd, gd = zd + (add.detach().double() if add is not None else 0), gy
    _close(y.detach(), yd.detach())
    y.backward(gy)
    zd.backward(_r16(gd))
    check_status()
    for got, want in ((x.grad, xd.grad), (w.grad, wd.grad)):
        _close(got, want)
    # the bias gradient is a sum of the bf16-rounded gradient
    _close(b.grad, bd.grad)
    if add is not None:
        assert torch.equal(add.grad, gy)


def test_block_with_hooks():
    """The residual block fuses only convolutions that nobody looks at."""
    import ferrum_b200 as fb
    from ferrum_b200.models import BasicBlock

    torch.manual_seed(0)
    block = BasicBlock(8, 16, 2, device=fb.Device.Cuda(0))
    x = torch.randn(2, 8, 14, 14, device="cuda")
    with fb.autocast():
        block(x).sum().backward()
    grads = [p.grad.clone() for p in block.torch_parameters()]
    seen = []
    hooks = [c.register_forward_hook(lambda m, i, o: seen.append(tuple(o.shape))) for c in (block.conv1, block.conv2)]
    for p in block.torch_parameters():
        p.grad = None
    with fb.autocast():
        got = block(x)
        loss = got.sum()
    got.detach().mul_(0.0)  # the output is the caller's
    loss.backward()
    assert seen == [(2, 16, 7, 7)] * 2
    for p, g in zip(block.torch_parameters(), grads):
        assert torch.equal(p.grad, g)
    for h in hooks:
        h.remove()


@pytest.mark.parametrize("k,pad,dil", [((3, 3), (-1, -2), (1, 1)), ((1, 1), (-1, 0), (1, 1)), ((2, 3), (1, -3), (2, 1))])
def test_negative_padding(k, pad, dil):
    """A crop, as long as the stride is 1."""
    import ferrum_b200 as fb
    from ferrum_b200 import nn
    from ferrum_b200.utils.runtime import check_status

    torch.manual_seed(1)
    conv = nn.Conv2d(8, 16, k, 1, pad, dil, device=fb.Device.Cuda(0))
    x = torch.randn(2, 8, 13, 17, device="cuda", requires_grad=True)
    with fb.autocast():
        y = conv(x)
    xd, wd, bd = (t.detach().double().requires_grad_(True) for t in (_r16(x.detach()), _r16(conv.weight.detach()), conv.bias))
    want = torch.nn.functional.conv2d(torch.nn.functional.pad(xd, (pad[1], pad[1], pad[0], pad[0])), wd, bd, 1, 0, dil)
    gy = torch.randn_like(y)
    y.backward(gy)
    want.backward(_r16(gy))
    check_status()
    for got, ref in ((y.detach(), want.detach()), (x.grad, xd.grad), (conv.weight.grad, wd.grad), (conv.bias.grad, bd.grad)):
        _close(got, ref)


def test_long_sequences():
    """Conv1d over more than 2^21 samples (an image of one row)."""
    import ferrum_b200 as fb
    from ferrum_b200 import nn
    from ferrum_b200.utils.runtime import check_status

    torch.manual_seed(2)
    conv = nn.Conv1d(1, 2, 5, 1, 2, device=fb.Device.Cuda(0))
    x = torch.randn(1, 1, 2 ** 21 + 77, device="cuda", requires_grad=True)
    with fb.autocast():
        y = conv(x)
    xd, wd, bd = (t.detach().double().requires_grad_(True) for t in (_r16(x.detach()), _r16(conv.weight.detach()), conv.bias))
    want = torch.nn.functional.conv1d(xd, wd, bd, 1, 2)
    gy = torch.randn_like(y)
    y.backward(gy)
    want.backward(_r16(gy))
    check_status()
    _close(y.detach(), want.detach()), _close(x.grad, xd.grad)
    # 64 partial sums of 2^15 products (about 2^7.5), 16 of them added at a time, truncated by 2^-23 of the sum so far: at
    # most 2^6 2^11 2^-23 2^7.5 = 2^1.5 in a gradient of about 2^10.5
    assert (conv.weight.grad.double() - wd.grad).norm() <= 2.0 ** -9 * wd.grad.norm()


def test_in_place_change_in_front_of_the_second_convolution():
    """A hook of conv2 may change what the block's ReLU wrote."""
    import ferrum_b200 as fb
    from ferrum_b200.models import BasicBlock

    torch.manual_seed(3)
    block = BasicBlock(8, 16, 2, device=fb.Device.Cuda(0))
    x = torch.randn(2, 8, 14, 14, device="cuda")

    def grads(hook):
        h = block.conv2.register_forward_pre_hook(hook)
        for p in block.torch_parameters():
            p.grad = None
        with fb.autocast():
            block(x).sum().backward()
        h.remove()
        return [p.grad.clone() for p in block.torch_parameters()]

    got = grads(lambda m, a: (a[0].mul_(0.5),))
    want = grads(lambda m, a: (a[0] * 0.5,))
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_filters_of_more_than_2_to_the_31():
    """Packing and folding alone, one channel padded to eight."""
    from ferrum_b200 import _lib

    lib, st, O = _lib.cuda(), torch.cuda.current_stream().cuda_stream, 2 ** 28 + 5
    w = torch.arange(O, device="cuda", dtype=torch.int32).remainder_(251).float()
    out = torch.full((O, 8), 3.0, device="cuda", dtype=torch.bfloat16)
    _lib.check(lib.fb_conv_pack_filters(w.data_ptr(), out.data_ptr(), O, 1, 1, 1, 1, 1, 1, 1, 8, 0, st), "fb_conv_pack_filters")
    assert torch.equal(out[:, 0].float(), w) and not out[:, 1:].any()
    del out
    part = torch.full((1, O, 8), 3.0, device="cuda")
    part[0, :, 0] = w
    dw = torch.full((O,), 7.0, device="cuda")
    _lib.check(lib.fb_conv_fold_wgrad(part.data_ptr(), dw.data_ptr(), 1, O, 1, 1, 1, 1, 1, 1, 1, 8, st), "fb_conv_fold_wgrad")
    assert torch.equal(dw, w)
    del part, dw
    torch.cuda.empty_cache()
