"""fp32 GEMM on the tensor cores: edges of its tiles, K splits and layouts against fp64.

Bound: the three dropped products are below 3 * 2^-26 of |a b|, a k-block of 64 adds six truncations per 16 products and
the k-blocks are added rounded to nearest; together below 5e-7 of the result's norm for zero-mean operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operand(rows, k, layout, g):
    if layout == "rows":                       # rows contiguous
        return torch.randn(k, rows, device="cuda", generator=g).t()
    if layout == "odd":                        # K contiguous, pitch not a multiple of 16 bytes
        return torch.randn(rows, k + 1, device="cuda", generator=g)[:, :k]
    return torch.randn(rows, k, device="cuda", generator=g)


@pytest.mark.parametrize("la,lb", [("k", "k"), ("k", "rows"), ("rows", "rows"), ("odd", "k"), ("rows", "odd")])
@pytest.mark.parametrize("M,N,K", [(1, 1, 33), (128, 64, 64), (129, 65, 65), (127, 10, 784), (300, 520, 129),
                                   (1, 4096, 512), (777, 1001, 333), (2048, 1280, 320), (4, 4, 5000)])
def test_layouts_and_edges(la, lb, M, N, K):
    from ferrum_b200.ops.gemm import gemm_f32
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = _operand(M, K, la, g), _operand(N, K, lb, g)
    bias = torch.randn(N, device="cuda", generator=g)
    ref = a.double() @ b.double().t() + bias.double()
    out = gemm_f32(a, b, bias=bias)
    check_status()
    assert (out.double() - ref).norm() <= 5e-7 * ref.norm() + 1e-6
    acc = torch.ones(M, N, device="cuda")
    gemm_f32(a, b, bias=bias, act="relu", out=acc, accumulate=True)
    assert (acc.double() - 1 - ref.clamp_min(0)).norm() <= 5e-7 * ref.norm() + 1e-5


def test_batched_strides():
    from ferrum_b200.ops import functional as F

    g = torch.Generator(device="cuda").manual_seed(3)
    q, k = (torch.randn(3, 197, 6, 64, device="cuda", generator=g).permute(0, 2, 1, 3) for _ in range(2))
    ref = 0.125 * (q.double() @ k.double().transpose(-1, -2))
    out = F.bmm_scaled(q, k.transpose(-1, -2), 0.125)
    assert (out.double() - ref).norm() <= 5e-7 * ref.norm()


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38, 1e-41])
def test_values_outside_the_split(value):
    from ferrum_b200.ops.gemm import gemm_f32

    g = torch.Generator(device="cuda").manual_seed(9)
    a, b = torch.rand(130, 100, device="cuda", generator=g), torch.rand(70, 100, device="cuda", generator=g)
    a[5, 7] = value
    b[3] *= 0.5
    ref, out = a.double() @ b.double().t(), gemm_f32(a, b).double()
    fine = torch.isfinite(ref.float())
    assert torch.equal(fine, torch.isfinite(out)) and torch.equal(ref.isnan(), out.isnan())
    assert (out - ref)[fine].abs().max() <= 1e-6 * ref[fine].abs().max()


@pytest.mark.parametrize("ea,eb", [(-120, 100), (100, -120), (-126, 90), (-140, 100),
                                   (-148, 110), (-60, -60), (100, -100), (60, 30), (115, -20), (55, 50)])
def test_operands_of_any_exponent(ea, eb):
    """The smallest operands decide the result, the largest leave the split: the bound is that of ordinary values of one
    sign (100 terms: a truncation per 16 products and k-block, or 100 roundings of a chain: below 2e-6)."""
    from ferrum_b200.ops.gemm import gemm_f32

    g = torch.Generator(device="cuda").manual_seed(11)
    a = torch.ldexp(1 + torch.rand(70, 100, device="cuda", generator=g), torch.tensor(ea, device="cuda"))
    b = torch.ldexp(1 + torch.rand(130, 100, device="cuda", generator=g), torch.tensor(eb, device="cuda"))
    ref, out = a.double() @ b.double().t(), gemm_f32(a, b).double()
    assert (out - ref).abs().max() <= 2e-6 * ref.abs().max()


@pytest.mark.parametrize("K", [33, 64, 100, 784, 4096])
def test_operands_of_one_sign(K):
    """Truncation is a bias that shows where all products have one sign: no further from fp64 than a chain of fp32
    multiply-adds (K / 2 roundings at random, and never below two roundings of the result)."""
    from ferrum_b200.ops.gemm import gemm_f32

    g = torch.Generator(device="cuda").manual_seed(K)
    a, b = torch.rand(300, K, device="cuda", generator=g), torch.rand(200, K, device="cuda", generator=g)
    ref = a.double() @ b.double().t()
    err = lambda o: ((o.double() - ref).norm() / ref.norm()).item()
    assert err(gemm_f32(a, b)) <= max(err(gemm_f32(a, b, simt=True)), 2.0 ** -23)


@pytest.mark.parametrize("lead_a,lead_b", [((3,), (3,)), ((), ()), ((2, 3), (3,)), ((3, 2, 2), (3, 2, 2))])
def test_scaled_products_of_other_ranks(lead_a, lead_b):
    """``bmm_scaled`` takes in fp32 what ``matmul`` takes."""
    from ferrum_b200.ops import functional as F

    g = torch.Generator(device="cuda").manual_seed(4)
    a, b = (torch.randn(*l, *s, device="cuda", generator=g) for l, s in ((lead_a, (5, 40)), (lead_b, (40, 7))))
    ref = 0.5 * (a.double() @ b.double())
    assert (F.bmm_scaled(a, b, 0.5).double() - ref).norm() <= 5e-7 * ref.norm()


@pytest.mark.parametrize("la", ["k", "rows", "odd"])
@pytest.mark.parametrize("M,N,K", [(5, 4, 33), (130, 12, 64), (31, 68, 100), (128, 132, 257), (96, 1028, 1030),
                                   (777, 1000, 333), (600, 1004, 520), (513, 904, 1030)])
def test_rows_of_b_by_quads(la, M, N, K):
    """B with its rows contiguous on 16-byte boundaries (read eight rows at a time) where the last eight are not whole or the
    last tile has no more of them, for each way in which A reaches tensor memory; the operand ends where the last row of K does.  Bound as above."""
    from ferrum_b200.ops.gemm import gemm_f32
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = _operand(M, K, la, g), _operand(N, K, "rows", g)
    ref = a.double() @ b.double().t()
    out = gemm_f32(a, b)
    check_status()
    assert (out.double() - ref).norm() <= 5e-7 * ref.norm() + 1e-6
    assert torch.equal(out, gemm_f32(a.contiguous(), b.contiguous()))  # the same sums, however the operands lie
