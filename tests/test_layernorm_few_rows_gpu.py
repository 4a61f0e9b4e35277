"""LayerNorm forward with a block per row: the same bits as a row gets among many (a warp per row), at both sides of the
line between the two and at widths with a partly filled last vector."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1024, 1032, 2048, 2056, 3000, 4096])
@pytest.mark.parametrize("rows", [1, 2, 296, 297])
def test_same_bits_as_among_many_rows(rows, cols):
    from ferrum_b200.ops import functional as F

    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(2000, cols, device="cuda", generator=g).bfloat16() * 3 + 1
    gamma, beta = (torch.randn(cols, device="cuda", generator=g) for _ in range(2))
    for ga, be in ((gamma, beta), (None, None)):
        few, many = F.layer_norm(x[:rows], ga, be, 1e-5), F.layer_norm(x, ga, be, 1e-5)
        assert torch.equal(few, many[:rows])
