"""LayerNorm(x + r) as one node against the addition and the normalisation as nodes of their own: the same arithmetic, so
the same bits forward; gradients too, the parameters' from partial sums in another order (2^-20 of their norm)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 256), (300, 264), (33, 1024), (513, 1032), (5, 4096), (9, 8192),
                                       (3, 8200), (4, 1001)])
def test_against_two_nodes(rows, cols, r_dtype):
    from ferrum_b200.ops import functional as F
    from ferrum_b200.utils.runtime import check_status

    got = []
    for fused in (True, False):
        g = torch.Generator(device="cuda").manual_seed(rows + cols)
        rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
        x, r = rand(2, rows, cols).requires_grad_(True), rand(2, rows, cols).to(r_dtype).requires_grad_(True)
        w, b = rand(cols).requires_grad_(True), rand(cols).requires_grad_(True)
        y = F.add_layer_norm(x, r, w, b) if fused else F.layer_norm(F.binary(x, r, "add"), w, b)
        with torch.no_grad():
            z = F.add_layer_norm(x, r, w, b)
        y.backward(rand(2, rows, cols))
        check_status()
        assert torch.equal(y.detach(), z)
        got.append((y.detach(), x.grad, r.grad, w.grad, b.grad))
    assert all(a.dtype == c.dtype and a.shape == c.shape for a, c in zip(*got))
    assert all(torch.equal(a, c) for a, c in zip(got[0][:3], got[1][:3]))
    for a, c in zip(got[0][3:], got[1][3:]):
        assert (a - c).norm() <= 2.0 ** -20 * c.norm()


@pytest.mark.parametrize("r_dtype", [torch.float32, torch.bfloat16])
def test_values_that_are_not_finite(r_dtype):
    from ferrum_b200.ops import functional as F

    got = []
    for fused in (True, False):
        g = torch.Generator(device="cuda").manual_seed(5)
        x, r, w = (torch.randn(*s, device="cuda", generator=g) for s in ((9, 264), (9, 264), (264,)))
        x[1, 3], r[4, 7], x[6, 0], r[6, 0] = float("inf"), float("nan"), float("inf"), float("-inf")
        x, r = x.requires_grad_(True), r.to(r_dtype).requires_grad_(True)
        y = F.add_layer_norm(x, r, w, None) if fused else F.layer_norm(F.binary(x, r, "add"), w, None)
        y.backward(torch.ones_like(y))
        got.append((y.detach(), x.grad, r.grad))
    for a, b in zip(*got):
        assert torch.equal(torch.isnan(a).any(1).nonzero().flatten().cpu(), torch.tensor([1, 4, 6]))
        assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))


def test_no_rows_have_empty_sums():
    from ferrum_b200 import _lib

    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream
    for added in (False, True):
        stats = torch.full((3, 24), float("nan"), device="cuda")
        if added:
            rc = lib.fb_add_layernorm_bwd(None, None, None, None, None, None, None, None, stats.data_ptr(), 0, 24, 1, st)
        else:
            rc = lib.fb_layernorm_bwd(None, None, None, None, None, None, None, None, stats.data_ptr(), 0, 24, 0, 0, 1, 2, st)
        assert rc == 0 and not stats.any()
