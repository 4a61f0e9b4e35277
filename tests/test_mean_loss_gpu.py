"""Mean losses at the edges of their launch forms: one cluster / whole grid, register rows / strided rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,bound", [(torch.float32, 4e-6), (torch.bfloat16, 8e-3)])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 37), (128, 10), (262, 1000), (263, 1000), (9, 264), (5, 4096), (7, 4104)])
def test_cross_entropy_and_nll(rows, cols, dtype, bound):
    """Gradients against fp64; the bound is a few roundings of the result's type (2^-24, 2^-9)."""
    from ferrum_b200 import nn

    g = torch.Generator(device="cuda").manual_seed(rows * 7 + cols)
    x = (3 * torch.randn(rows, cols, device="cuda", generator=g)).to(dtype).requires_grad_(True)
    t = torch.randint(0, cols, (rows,), device="cuda", generator=g)
    for fn, ref in ((nn.cross_entropy, torch.nn.functional.cross_entropy), (nn.nll_loss, torch.nn.functional.nll_loss)):
        xd = x.detach().double().requires_grad_(True)
        want = ref(xd, t)
        (want * 3).backward()
        x.grad = None
        loss = fn(x, t)
        (loss * 3).backward()
        assert abs(loss.item() - want.item()) <= bound * max(1.0, abs(want.item()))
        assert (x.grad.double() - xd.grad).norm() <= bound * xd.grad.norm() + 1e-12


@pytest.mark.parametrize("n", [1, 5, 262144, 262145, 1 << 21])
def test_elementwise_loss_sum(n):
    """n additions in blocks of a few thousand: relative error below 1e-5 for sums of positive terms."""
    from ferrum_b200 import nn

    g = torch.Generator(device="cuda").manual_seed(n)
    p, t = (torch.randn(n, device="cuda", generator=g) for _ in range(2))
    want = ((p.double() - t.double()) ** 2).mean().item()
    assert abs(nn.mse_loss(p, t).item() - want) <= 1e-5 * want


def test_nll_targets_of_another_number_or_device():
    """More targets than rows and targets on the CPU are errors; rows past the last target add nothing to the sum."""
    from ferrum_b200 import nn

    lp = torch.log_softmax(torch.randn(6, 5, device="cuda"), -1)
    t = torch.randint(0, 5, (8,), device="cuda")
    for bad in (t, t[:6].cpu()):
        for fn in (nn.nll_loss, nn.cross_entropy_loss):
            with pytest.raises((RuntimeError, ValueError)):
                fn(lp, bad)
    want = -lp[:4].gather(1, t[:4, None]).sum() / 6
    assert abs(nn.nll_loss(lp, t[:4]).item() - want.item()) < 1e-6


@pytest.mark.parametrize("bad", [-1, 5])
@pytest.mark.parametrize("rows", [6, 300000])
def test_nll_class_out_of_range(rows, bad):
    """Reported in the status block and by the loss itself; nothing is read outside the row."""
    from ferrum_b200 import nn
    from ferrum_b200.utils.runtime import DeviceStatusError, check_status

    lp = torch.log_softmax(torch.randn(rows, 5, device="cuda"), -1).requires_grad_(True)
    t = torch.randint(0, 5, (rows,), device="cuda")
    t[rows // 2] = bad
    check_status()
    loss = nn.nll_loss(lp, t)
    with pytest.raises(DeviceStatusError, match="bounds_violation"):
        check_status()
    assert loss.isnan()
    loss.backward()
    check_status()
