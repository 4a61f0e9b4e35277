"""A residual block as one node against the same block as nodes of its own (a hook that does nothing keeps it from being one):
the same products of the same operands, so the bits are the same.  The epilogues that only the one node uses, and the block as a
whole, against plain PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(block, x, need_x, change):
    import ferrum_b200 as fb

    x = x.clone().requires_grad_(need_x)
    weights = [c.weight for c in (block.conv1, block.conv2, block.downsample) if c is not None and c.weight.requires_grad]
    for p in weights:
        p.grad = None
    with fb.autocast():
        y = block(x)
    out = y.detach().clone()
    if change:
        y = y.add_(1.0)
    g = torch.randn(y.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    if y.requires_grad:
        y.backward(g)
    return [out] + [p.grad.clone() for p in weights] + ([x.grad] if need_x else [])


@pytest.mark.parametrize("cin,cout,stride,size,batch", [(8, 8, 1, 9, 2), (16, 24, 2, 15, 3), (64, 64, 1, 28, 2), (5, 16, 1, 12, 2),
                                                        (24, 16, 2, 14, 1), (3, 136, 2, 7, 5), (8, 12, 1, 8, 2)])
@pytest.mark.parametrize("value", [None, float("nan"), float("inf")])
def test_bits(cin, cout, stride, size, batch, value):
    import ferrum_b200 as fb
    from ferrum_b200.models import BasicBlock
    from ferrum_b200.utils.runtime import check_status

    fb.manual_seed(cin + cout)
    block = BasicBlock(cin, cout, stride, device=fb.Device.Cuda(0))
    x = torch.randn(batch, cin, size, size, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    if value is not None:
        x[0, 0, 3, 3] = value
    one = [_run(block, x, need_x, change) for need_x, change in ((True, False), (False, False), (True, True))]
    with torch.no_grad(), fb.autocast():
        plain = block(x)
    hook = block.conv2.register_forward_hook(lambda *a: None)
    several = [_run(block, x.detach(), need_x, change) for need_x, change in ((True, False), (False, False), (True, True))]
    hook.remove()
    check_status()
    same = lambda a, b: torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
    assert same(plain, one[0][0])
    for a, b in zip(one, several):
        assert len(a) == len(b) and all(same(s, t) for s, t in zip(a, b))


def test_which_node():
    import ferrum_b200 as fb
    from ferrum_b200.models import BasicBlock

    x = torch.randn(2, 16, 10, 10, device="cuda", requires_grad=True)
    for cout, stride in ((16, 1), (24, 2), (24, 1)):
        block = BasicBlock(16, cout, stride, device=fb.Device.Cuda(0))
        with fb.autocast():
            assert block(x).grad_fn.name() == "FerrumConvBlockBackward"
            for conv in (block.conv1, block.conv2, block.downsample):
                if conv is not None:
                    hook = conv.register_forward_hook(lambda *a: None)
                    assert block(x).grad_fn.name() != "FerrumConvBlockBackward"
                    hook.remove()
            assert block(x.bfloat16()).grad_fn.name() != "FerrumConvBlockBackward"
        assert block(x).grad_fn.name() != "FerrumConvBlockBackward"  # fp32
    with pytest.raises(Exception):
        with fb.autocast():
            BasicBlock(16, 16, 1, device=fb.Device.Cuda(0))(x[:, :8])


def _conv(*args):
    from ferrum_b200 import nn

    return nn.Conv2d.with_config(*args, 1, False).to("cuda")  # one group, no bias


def _same(a, b):
    return len(a) == len(b) and all(torch.equal(s, t) for s, t in zip(a, b))


# channels, size, then kernel, stride, padding and dilation of each convolution
GEOMETRIES = {
    "5x5 down": (8, 16, 11, (5, 2, 2, 1), (5, 1, 2, 1), (1, 2, 0, 1)),
    "dilated": (8, 8, 11, (3, 1, 2, 2), (3, 1, 4, 4), None),
    "1x1": (16, 16, 9, (1, 1, 0, 1), (1, 1, 0, 1), None),
    "wide shortcut": (8, 24, 13, (3, 2, 1, 1), (3, 1, 1, 1), (3, 2, 1, 1)),
    "stride 3": (5, 16, 14, (3, 3, 1, 1), (3, 1, 1, 1), (1, 3, 0, 1)),
    "negative padding": (8, 16, 12, (3, 1, -1, 1), (3, 1, 2, 1), (3, 1, 0, 1)),
    "grows and shrinks": (8, 8, 10, (3, 1, 2, 1), (3, 1, 0, 1), None),
    "shortcut of stride 1": (12, 20, 9, (3, 1, 1, 1), (3, 1, 1, 1), (1, 1, 0, 1)),
}


def _block(cin, cout, first, second, short):
    import ferrum_b200 as fb
    from ferrum_b200.models import BasicBlock

    mid = cout if cout % 8 == 0 else 16
    block = BasicBlock(cin, cout, 1, device=fb.Device.Cuda(0))
    block.conv1, block.conv2 = _conv(cin, mid, *first), _conv(mid, cout, *second)
    block.downsample = None if short is None else _conv(cin, cout, *short)
    return block


@pytest.mark.parametrize("name", GEOMETRIES)
def test_geometries(name):
    import ferrum_b200 as fb
    from ferrum_b200.utils.runtime import check_status

    cin, cout, size, *convs = GEOMETRIES[name]
    fb.manual_seed(3)
    block = _block(cin, cout, *convs)
    x = torch.randn(3, cin, size, size, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    with fb.autocast():
        assert block(x).grad_fn.name() == "FerrumConvBlockBackward"
    one = _run(block, x, True, False)
    hook = block.conv2.register_forward_hook(lambda *a: None)
    several = _run(block, x, True, False)
    hook.remove()
    check_status()
    assert _same(one, several)
    # PyTorch in 64 bits with the same roundings to bf16: sums in 32 bits may round another way there, a unit of 2^-8 in few values
    low = lambda t: t.detach().bfloat16().double()
    w1, w2, wd = (None if c is None else low(c.weight) for c in (block.conv1, block.conv2, block.downsample))
    kw = [None if c is None else dict(stride=c[1], padding=max(c[2], 0), dilation=c[3]) for c in convs]
    cut = max(-convs[0][2], 0)
    conv, into, over = torch.nn.functional.conv2d, torch.nn.grad.conv2d_input, torch.nn.grad.conv2d_weight
    z1 = low(x)[:, :, cut:size - cut, cut:size - cut]
    z2 = low(conv(z1, w1, **kw[0]).relu())
    y = (conv(z2, w2, **kw[1]) + (x.double() if wd is None else conv(low(x), wd, **kw[2]))).relu()
    g = torch.randn(y.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).double() * (y > 0)
    g1 = low(into(z2.shape, w2, low(g), **kw[1]) * (z2 > 0))
    dx = torch.nn.functional.pad(into(z1.shape, w1, g1, **kw[0]), [cut] * 4)
    dx = dx + (g if wd is None else into(x.shape, wd, low(g), **kw[2]))
    want = [y, over(z1, w1.shape, g1, **kw[0]), over(z2, w2.shape, low(g), **kw[1])]
    want += ([] if wd is None else [over(low(x), wd.shape, low(g), **kw[2])]) + [dx]
    assert len(one) == len(want)
    for got, ref in zip(one, want):
        assert (got - ref).norm() <= 2.0 ** -9 * ref.norm()


@pytest.mark.parametrize("frozen", [("conv1",), ("conv2",), ("downsample",), ("conv1", "conv2"), ("conv1", "conv2", "downsample")])
@pytest.mark.parametrize("need_x", [True, False])
def test_frozen_filters(frozen, need_x):
    import ferrum_b200 as fb
    from ferrum_b200.models import BasicBlock

    fb.manual_seed(4)
    block = BasicBlock(8, 16, 2, device=fb.Device.Cuda(0))
    for name in frozen:
        getattr(block, name).weight.requires_grad_(False)
    x = torch.randn(2, 8, 11, 11, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    one = _run(block, x, need_x, False)
    block.conv2.register_forward_hook(lambda *a: None)
    assert _same(one, _run(block, x, need_x, False))


def test_filters_shared_by_both_convolutions():
    import ferrum_b200 as fb
    from ferrum_b200.models import BasicBlock

    fb.manual_seed(6)
    block = BasicBlock(16, 16, 1, device=fb.Device.Cuda(0))
    block.conv2.weight = block.conv1.weight
    x = torch.randn(2, 16, 9, 9, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7))
    one = _run(block, x, True, False)
    block.conv2.register_forward_hook(lambda *a: None)
    assert _same(one, _run(block, x, True, False))


@pytest.mark.parametrize("B,H,W,C,O,k", [(2, 9, 7, 8, 16, 3), (1, 5, 5, 16, 5, 1), (3, 28, 28, 64, 128, 3), (2, 12, 33, 24, 72, 5)])
def test_epilogues(B, H, W, C, O, k):
    """ReLU, a mask and a result that is added to, of sums in 32 bits of C k^2 products: 2^-24 of the magnitudes per product at
    most, and half a unit of bf16 (2^-9) where the result is that."""
    from ferrum_b200 import _lib
    from ferrum_b200.utils.runtime import check_status, status_ptr

    g = torch.Generator(device="cuda").manual_seed(O)
    new = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, old, mask = new(B, H, W, C).bfloat16(), new(O, k * k, C).bfloat16(), new(B, H, W, O), new(B, H, W, O).bfloat16()
    mask.view(-1)[::3] = 0
    lib, st, pad = _lib.cuda(), torch.cuda.current_stream().cuda_stream, k // 2
    xd, wd = x.double().permute(0, 3, 1, 2), w.double().view(O, k, k, C).permute(0, 3, 1, 2)
    want, size = (torch.nn.functional.conv2d(a, b, padding=pad).permute(0, 2, 3, 1) for a, b in ((xd, wd), (xd.abs(), wd.abs())))
    tol = C * k * k * 2.0 ** -24 * size + 1e-30

    def run(y, m=None, act=0, beta=0):
        _lib.check(lib.fb_conv_igemm_epilogue(x.data_ptr(), w.data_ptr(), y.data_ptr(), None, None if m is None else m.data_ptr(), B,
                                              H, W, C, O, k, k, pad, pad, 1, 1, O, int(y.dtype == torch.bfloat16), act, beta,
                                              status_ptr(), st), "conv")
        check_status()
        return y.double()

    assert ((run(old.clone(), beta=1) - old - want).abs() <= tol + 2.0 ** -23 * (old.abs() + want.abs())).all()
    low = torch.full_like(mask, float("nan"))
    assert ((run(low, act=1) - want.clamp(min=0)).abs() <= tol + 2.0 ** -8 * want.abs()).all()
    got = run(torch.full_like(mask, float("nan")), m=mask)
    assert ((got - want).abs() <= tol + 2.0 ** -8 * want.abs())[mask > 0].all() and not got[~(mask > 0)].any()
    assert lib.fb_conv_igemm_epilogue(x.data_ptr(), w.data_ptr(), old.data_ptr(), None, mask.data_ptr(), B, H, W, C, O, k, k, pad, pad,
                                      1, 1, O, 0, 0, 0, status_ptr(), st) == -1  # a mask of an fp32 result
