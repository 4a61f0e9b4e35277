"""A residual block as one node against the same block as nodes of its own (a hook that does nothing keeps it from being one):
the same products of the same operands, so the bits are the same."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(block, x, need_x, change):
    import ferrum_b200 as fb

    x = x.clone().requires_grad_(need_x)
    weights = [c.weight for c in (block.conv1, block.conv2, block.downsample) if c is not None]
    for p in weights:
        p.grad = None
    with fb.autocast():
        y = block(x)
    out = y.detach().clone()
    if change:
        y = y.add_(1.0)
    g = torch.randn(y.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
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
