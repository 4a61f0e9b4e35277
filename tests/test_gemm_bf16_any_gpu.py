"""bf16 GEMM on operands that a TMA map cannot describe: tile edges, K splits, alignments and layouts against fp64.

Bound: products of bf16 numbers are exact in fp32, a k-block of 64 adds four truncated sums and the k-blocks are added
rounded to nearest: below 5e-7 of the result's norm for zero-mean operands; a bf16 result adds 2^-9."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operand(rows, k, layout, g):
    if layout == "rows":     # rows contiguous, odd pitch
        return torch.randn(k, rows + 1, device="cuda", generator=g).bfloat16()[:, 1:].t()
    if layout == "odd":      # K contiguous at an odd address, any pitch
        return torch.randn(rows * k + 3, device="cuda", generator=g).bfloat16()[3:].view(rows, k)
    if layout == "even":     # 16-byte aligned rows
        return torch.randn(rows, -(-k // 8) * 8, device="cuda", generator=g).bfloat16()[:, :k]
    return torch.randn(rows, 2 * k, device="cuda", generator=g).bfloat16()[:, ::2]  # no unit stride


@pytest.mark.parametrize("la,lb", [("odd", "odd"), ("odd", "rows"), ("rows", "rows"), ("even", "odd"), ("odd", "step")])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (128, 64, 64), (129, 65, 65), (127, 10, 771), (300, 520, 129),
                                   (1, 4095, 513), (777, 1001, 333), (2048, 1280, 321), (4, 4, 5001)])
def test_layouts_and_edges(la, lb, M, N, K):
    from ferrum_b200 import _lib
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = _operand(M, K, la, g), _operand(N, K, lb, g)
    bias = torch.randn(N, device="cuda", generator=g)
    ref = a.double() @ b.double().t() + bias.double()
    out = torch.full((M, N), 2.0, device="cuda")
    _lib.native().gemm_nt(a, b, bias, 1, out, True, False)   # relu, added to what is there
    check_status()
    assert (out.double() - 2 - ref.clamp_min(0)).norm() <= 5e-7 * (ref.norm() + 2 * (M * N) ** 0.5) + 1e-6
    low = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    _lib.native().gemm_nt(a, b, bias, 0, low, False, False)
    assert (low.double() - ref).norm() <= 2.0 ** -8 * ref.norm()


@pytest.mark.parametrize("la,lb", [("rows", "rows"), ("rows", "even"), ("odd", "odd"), ("odd", "even"), ("step", "rows"),
                                   ("flat", "flat"), ("flat", "even")])
@pytest.mark.parametrize("M,N,K", [(2049, 2049, 1024), (1001, 1200, 4096), (1601, 1603, 1000), (513, 333, 8192), (1001, 2000, 64)])
def test_large_products_of_aligned_reduction(la, lb, M, N, K):
    """Sizes where unaligned operands are copied first (the last one is not): the persistent kernels' bits, whose tensor
    core truncates K / 16 times: K / 16 * 2^-23 of the norm."""
    from ferrum_b200 import _lib
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    make = lambda rows, l: (torch.randn(K, rows, device="cuda", generator=g).bfloat16().t() if l == "flat"
                            else _operand(rows, K, l, g))
    a, b = make(M, la), make(N, lb)
    bias = torch.randn(N, device="cuda", generator=g)
    ref = a.double() @ b.double().t() + bias.double()
    bound = (K / 16 * 2.0 ** -23 + 1e-6)
    out = torch.full((M, N), 2.0, device="cuda")
    _lib.native().gemm_nt(a, b, bias, 1, out, True, False)
    check_status()
    assert (out.double() - 2 - ref.clamp_min(0)).norm() <= bound * (ref.norm() + 2 * (M * N) ** 0.5)
    low = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    _lib.native().gemm_nt(a, b, bias, 0, low, False, False)
    assert (low.double() - ref).norm() <= 2.0 ** -8 * ref.norm()
    if M * N > 2e6 and "step" not in (la, lb):
        aligned = torch.empty_like(low)
        _lib.native().gemm_nt(a.contiguous().clone(), b.contiguous().clone(), bias, 0, aligned, False, False)
        assert torch.equal(aligned, low)
