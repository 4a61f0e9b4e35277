"""LayerNorm over rows of any width, both directions, at the edges of the tiles, against fp64.

Bounds: fp32 sums of up to 8193 terms, two passes: 2e-6 of the norm; bf16 results and gradients round once more (2^-8 of
the norm covers an output rounding of 2^-9 and that of the GELU's fast evaluation)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 33), (130, 63), (7, 65), (900, 256), (5, 255), (64, 257), (700, 512),
                                       (777, 1001), (1500, 1024), (9, 1023), (4, 1025), (6, 2047), (300, 2048), (5, 2049),
                                       (3, 4095), (2, 4097), (3, 8191), (2, 8193),
                                       # where the rows that are held in registers end
                                       (888, 129), (889, 129), (1184, 127), (1185, 127), (593, 1793), (2369, 1795),
                                       (444, 2049), (445, 2049), (593, 4095), (444, 257), (445, 257), (593, 1025), (1185, 1025), (149, 4097),
                                       (593, 4097)])
@pytest.mark.parametrize("pre", [None, "gelu"])
def test_against_fp64(rows, cols, dtype, pre):
    from ferrum_b200.ops import functional as F
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, gy = rand(rows, cols).to(dtype), rand(rows, cols).to(dtype)
    w, b = rand(cols), rand(cols)
    leaves = [t.clone().requires_grad_(True) for t in (x, w, b)]
    exact = [t.double().requires_grad_(True) for t in (x, w, b)]
    y = F.layer_norm(leaves[0], leaves[1], leaves[2], 1e-5, pre)
    y.backward(gy)
    z = torch.nn.functional.gelu(exact[0], approximate="tanh") if pre else exact[0]
    want = torch.nn.functional.layer_norm(z, (cols,), exact[1], exact[2], 1e-5)
    want.backward(gy.double())
    check_status()
    tol = 2e-6 if dtype is torch.float32 else 2.0 ** -8
    assert (y.double() - want).norm() <= tol * want.norm() + 1e-6
    # a row of one column has no gradient; next to none there, absolute
    for got, ref in zip(leaves, exact):
        assert (got.grad.double() - ref.grad).norm() <= 2 * tol * ref.grad.norm() + 1e-5 * rows ** 0.5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(5, 33), (600, 257), (889, 129), (593, 1001), (20, 4097)])
def test_values_that_are_not_finite(rows, cols, dtype):
    """A row with an infinity or a NaN is NaN; the others keep their bits."""
    from ferrum_b200.ops import functional as F

    g = torch.Generator(device="cuda").manual_seed(cols)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    base, gy, w = rand(rows, cols).to(dtype), rand(rows, cols).to(dtype), rand(cols)

    def run(x):
        x = x.clone().requires_grad_(True)
        y = F.layer_norm(x, w, None)
        y.backward(gy)
        return y.detach(), x.grad

    clean = run(base)
    others = torch.arange(rows, device="cuda") != rows // 2
    for value in (float("inf"), float("nan")):
        x = base.clone()
        x[rows // 2, cols - 1] = value
        for got, want in zip(run(x), clean):
            assert torch.isnan(got[rows // 2]).all() and torch.equal(got[others], want[others])
