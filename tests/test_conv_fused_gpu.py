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


@pytest.mark.parametrize("C,stride", [(8, 1), (65, 1), (3, 2)])
@pytest.mark.parametrize("fused", ["relu", "add"])
def test_values_that_are_not_finite(C, stride, fused):
    """The bits of the convolution and the fused op as two nodes, in both directions; a value spoils its own windows, which
    strides round up to a multiple of themselves (with zeros as filter taps)."""
    import ferrum_b200 as fb
    from ferrum_b200.ops import functional as F

    g = torch.Generator(device="cuda").manual_seed(C)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    base, w = rand(2, C, 9, 10), rand(6, C, 3, 3)
    s = (stride, stride)
    with fb.autocast(), torch.no_grad():
        clean = F.conv2d_igemm(base, w, None, (1, 1), (1, 1), s)
    add, gy = rand(*clean.shape), rand(*clean.shape)
    for value in (float("inf"), float("nan")):
        x = base.clone()
        x[1, C - 1, 4, 5] = value
        results = []
        for one in (True, False):
            leaves = [t.clone().requires_grad_(True) for t in (x, w, add)]
            with fb.autocast():
                if one:
                    y = F.conv2d_igemm(leaves[0], leaves[1], None, (1, 1), (1, 1), s,
                                       leaves[2] if fused == "add" else None, "relu" if fused == "relu" else None)
                else:
                    z = F.conv2d_igemm(leaves[0], leaves[1], None, (1, 1), (1, 1), s)
                    y = F.unary(z, "relu") if fused == "relu" else F.binary(z, leaves[2], "add")
            y.backward(gy)
            results.append([y.detach()] + [t.grad for t in leaves if t.grad is not None])
        for a, b in zip(*results):
            assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
        with fb.autocast(), torch.no_grad():
            y = F.conv2d_igemm(x, w, None, (1, 1), (1, 1), s)
        k = -(-3 // stride) * stride
        bad = torch.nn.functional.pad((~torch.isfinite(x)).float().amax(1, keepdim=True), (1, k - 2, 1, k - 2))
        hit = torch.nn.functional.max_pool2d(bad, k, stride)[:, :, :y.shape[2], :y.shape[3]].bool().expand_as(y)
        assert torch.equal(~torch.isfinite(y), hit) and torch.equal(y[~hit], clean[~hit])


@pytest.mark.parametrize("shape", range(8))
def test_layouts(shape):
    """The layout kernels against the same arrangements in plain torch: exact but for the rounding to bf16, padding zero."""
    from ferrum_b200 import _lib

    from tests import _conv_s2d as s2d

    B, C, O, H, W, k, s, p = s2d.SHAPES[shape]
    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream
    x, w = torch.randn(B, C, H, W, device="cuda"), torch.randn(O, C, *k, device="cuda")
    Ho, Wo, k2h, k2w, Hz, Wz, eh, ew, Cz = s2d.geometry(x.shape, w.shape, s, p)
    sizes, bf = (B, C, H, W, *s, eh, ew, *p, Hz, Wz), dict(device="cuda", dtype=torch.bfloat16)
    mask = torch.randn_like(x)
    for m in (None, mask):
        z = torch.full((B, Hz, Wz, Cz), 3.0, **bf)
        _lib.check(lib.fb_conv_pack_input(x.data_ptr(), None if m is None else m.data_ptr(), z.data_ptr(), *sizes, Cz, st), "x")
        assert torch.equal(z, s2d.pack_input(x if m is None else torch.where(m > 0, x, 0.0), w.shape, s, p).bfloat16())
    filters = s2d.pack_filters(w, s, Cz)
    packed, Op = torch.full(filters.shape, 3.0, **bf), -(-O // 8) * 8
    _lib.check(lib.fb_conv_pack_filters(w.data_ptr(), packed.data_ptr(), O, C, *k, *s, eh, ew, Cz, 0, st), "w")
    assert torch.equal(packed, filters.bfloat16())
    turned = torch.full((eh * ew * C, k2h * k2w, Op), 3.0, **bf)
    _lib.check(lib.fb_conv_pack_filters(w.data_ptr(), turned.data_ptr(), O, C, *k, *s, eh, ew, Op, 1, st), "w turned")
    assert torch.equal(turned[..., :O], filters[..., :eh * ew * C].flip(1).permute(2, 1, 0).bfloat16())
    assert not turned[..., O:].any()
    part = torch.randn(3, *filters.shape, device="cuda")
    dw = torch.full_like(w, 7.0)
    _lib.check(lib.fb_conv_fold_wgrad(part.data_ptr(), dw.data_ptr(), 3, O, C, *k, *s, eh, ew, Cz, st), "dw")
    assert torch.equal(s2d.pack_filters(dw, s, Cz), torch.where(s2d.pack_filters(torch.ones_like(w), s, Cz) > 0,
                                                                part[0] + part[1] + part[2], 0.0))
    back = torch.full_like(x, 7.0)
    dz = torch.randn(B, Hz, Wz, eh * ew * C, device="cuda")
    _lib.check(lib.fb_s2d_nhwc_to_nchw_f32(dz.data_ptr(), back.data_ptr(), *sizes, eh * ew * C, st), "dx")
    reach = s2d.pack_input(torch.ones_like(x), w.shape, s, p)[..., :eh * ew * C] > 0
    assert torch.equal(s2d.pack_input(back, w.shape, s, p)[..., :eh * ew * C], torch.where(reach, dz, 0.0))
    # every value of z arrives once, the pixels that no window reaches are zero
    assert back.count_nonzero() == reach.sum()


@pytest.mark.parametrize("C,H,W,k,s,p", [(3, 2, 4, (3, 3), (2, 2), (1, 1)), (66, 3, 132, (3, 3), (2, 2), (1, 1)),
                                         (64, 2, 64, (5, 5), (3, 3), (2, 2)), (16, 3, 128, (3, 3), (2, 2), (0, 3)),
                                         (65, 6, 22, (3, 3), (1, 1), (0, 0)), (8, 5, 60, (4, 4), (4, 4), (3, 2))])
@pytest.mark.parametrize("off", [0, 1])
def test_layouts_by_quads_of_pixels(C, H, W, k, s, p, off):
    """Rows of whole quads, on 16-byte boundaries or one element behind (read one by one); tiles with an odd first column."""
    from ferrum_b200 import _lib

    from tests import _conv_s2d as s2d

    lib, st, B = _lib.cuda(), torch.cuda.current_stream().cuda_stream, 2
    x, m = (torch.randn(B * C * H * W + 1, device="cuda")[off:][:B * C * H * W].view(B, C, H, W) for _ in range(2))
    Ho, Wo, k2h, k2w, Hz, Wz, eh, ew, Cz = s2d.geometry(x.shape, (1, C, *k), s, p)
    for mask in (None, m):
        z = torch.full((B, Hz, Wz, Cz), 3.0, device="cuda", dtype=torch.bfloat16)
        _lib.check(lib.fb_conv_pack_input(x.data_ptr(), None if mask is None else m.data_ptr(), z.data_ptr(), B, C, H, W, *s,
                                          eh, ew, *p, Hz, Wz, Cz, st), "x")
        assert torch.equal(z, s2d.pack_input(x if mask is None else torch.where(m > 0, x, 0.0), (1, C, *k), s, p).bfloat16())
    for P in (H * W, H * W + 2):
        src, add, y = torch.randn(B, P, C + 3, device="cuda"), *(torch.randn(B * C * P + 1, device="cuda") for _ in range(2))
        add, y = (t[off:][:B * C * P].view(B, C, P) for t in (add, y))
        for a, relu in ((None, 0), (add, 1)):
            _lib.check(lib.fb_nhwc_to_nchw_f32(src.data_ptr(), None if a is None else a.data_ptr(), y.data_ptr(), B, C, P, C + 3,
                                               relu, st), "y")
            want = src[..., :C].transpose(1, 2) + (0 if a is None else a)
            assert torch.equal(y, want.relu() if relu else want)
