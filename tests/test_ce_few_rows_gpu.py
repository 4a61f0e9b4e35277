"""Cross-entropy around the row counts where the split over the chip changes (24 / 25 blocks of one row for wide rows, of
eight rows for others: 192 / 193) and at multiples of the SM count; odd and even class counts, against fp64 (fp32: 1e-6;
bf16 logits: their gradient rounds to 2^-9)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows", [1, 24, 25, 127, 148, 149, 192, 193, 296, 297, 592, 593, 777, 1184, 1185, 2369])
@pytest.mark.parametrize("classes", [2, 37, 40, 512, 1001])
def test_loss_and_gradient(rows, classes, dtype):
    import ferrum_b200.nn as nn
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(rows + classes)
    x = torch.randn(rows, classes, device="cuda", generator=g).to(dtype)
    t = torch.randint(0, classes, (rows,), device="cuda", generator=g)
    a, e = x.clone().requires_grad_(True), x.double().requires_grad_(True)
    loss = nn.cross_entropy(a, t)
    loss.backward()
    want = torch.nn.functional.cross_entropy(e, t)
    want.backward()
    check_status()
    assert abs(float(loss) - float(want)) <= 2e-6 * abs(float(want)) + 1e-6
    assert (a.grad.double() - e.grad).norm() <= (1e-6 if dtype is torch.float32 else 2.0 ** -8) * e.grad.norm()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,classes", [(24, 37), (193, 37), (25, 1001), (193, 1000)])
def test_values_that_are_not_finite(rows, classes, dtype):
    """An infinite or NaN logit stays in its row: the loss is what fp64 says, the other rows' gradients are untouched."""
    import ferrum_b200.nn as nn

    g = torch.Generator(device="cuda").manual_seed(rows)
    base = torch.randn(rows, classes, device="cuda", generator=g).to(dtype)
    t = torch.randint(0, classes - 1, (rows,), device="cuda", generator=g)

    def grad(x):
        a = x.clone().requires_grad_(True)
        loss = nn.cross_entropy(a, t)
        loss.backward()
        return loss.detach(), a.grad

    _, clean = grad(base)
    for value in (float("-inf"), float("inf"), float("nan")):
        x = base.clone()
        x[rows // 2, classes - 1] = value
        loss, dx = grad(x)
        want = torch.nn.functional.cross_entropy(x.double(), t)
        if value == float("-inf"):
            assert torch.isfinite(dx).all() and abs(float(loss) - float(want)) <= 2e-6 * abs(float(want)) + 1e-6
        else:
            assert not torch.isfinite(loss) and not torch.isfinite(want) and torch.isnan(dx[rows // 2]).any()
        others = torch.arange(rows, device="cuda") != rows // 2
        assert torch.equal(dx[others], clean[others])
