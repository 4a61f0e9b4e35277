"""bf16 GEMM with the K splits of a tile in a cluster: every tile shape at its edges, both layouts, against fp64.

Bound: products of bf16 numbers are exact in fp32; the tensor core truncates where it adds, at most K / 16 times within
a split: K / 16 * 2^-23 of the result's norm, plus 1e-6; a bf16 result adds 2^-9."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operand(rows, k, mn, g):
    pad = lambda n: -(-n // 8) * 8
    if mn:
        return torch.randn(k, pad(rows), device="cuda", generator=g).bfloat16()[:, :rows].t()
    return torch.randn(rows, pad(k), device="cuda", generator=g).bfloat16()[:, :k]


def _call(a, b, out, out2, bias, act, beta, tile):
    from ferrum_b200 import _lib
    from ferrum_b200.ops.gemm import _major
    from ferrum_b200.utils import runtime as rt

    (a_mn, lda), (b_mn, ldb) = _major(a), _major(b)
    p = lambda t: None if t is None else t.data_ptr()
    _lib.check(_lib.cuda().fb_gemm_bf16_splitk(
        p(a), p(b), p(out), p(out2), p(bias), a.shape[0], b.shape[0], a.shape[1], lda, ldb, out.stride(0), a_mn, b_mn,
        int(out.dtype == torch.bfloat16), act, beta, tile, rt.status_ptr(), torch.cuda.current_stream().cuda_stream),
        "fb_gemm_bf16_splitk")


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("tile,M,N,K", [(16, 1, 1, 8), (16, 16, 4096, 4096), (16, 17, 130, 513), (32, 31, 1000, 1024),
                                        (64, 64, 128, 64), (64, 33, 257, 2047), (192, 128, 64, 128),
                                        (192, 129, 65, 4103), (256, 511, 1001, 640), (256, 257, 129, 65)])
def test_tiles(tile, M, N, K, a_mn, b_mn):
    from ferrum_b200.ops.gemm import ACT
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b = _operand(M, K, a_mn, g), _operand(N, K, b_mn, g)
    bias = torch.randn(N, device="cuda", generator=g)
    ref = a.double() @ b.double().t() + bias.double()
    bound = K / 16 * 2.0 ** -23 + 1e-6
    out = torch.full((M, N + 3), 2.0, device="cuda")[:, :N]
    _call(a, b, out, None, bias, ACT["relu"], 1, tile)
    check_status()
    assert (out.double() - 2 - ref.clamp_min(0)).norm() <= bound * (ref.norm() + 2 * (M * N) ** 0.5)
    low, der = (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    _call(a, b, low, der, bias, ACT["sigmoid"], 0, tile)
    s = ref.sigmoid()
    # the rounding of z (its norm times the bound) passes through a slope of at most 1 / 4
    assert (low.double() - s).norm() <= 2.0 ** -8 * s.norm() + bound * ref.norm()
    assert (der.double() - s * (1 - s)).norm() <= 2.0 ** -8 * s.norm() + bound * ref.norm()


def test_linear_of_few_rows_in_either_grad_mode():
    import ferrum_b200 as fb
    from ferrum_b200 import nn

    torch.manual_seed(2)
    lin = nn.Linear(4096, 520, device=fb.Device.Cuda(0))
    x = torch.randn(5, 4096, device="cuda")
    with fb.autocast():
        y = lin(x)
        with fb.no_grad():
            z = lin(x)
    ref = x.bfloat16().double() @ lin.weight.detach().bfloat16().double().t() + lin.bias.detach().double()
    assert torch.equal(y.detach(), z)
    for out in (y, z):
        assert (out.detach().double() - ref).norm() <= 2.0 ** -8 * ref.norm()
