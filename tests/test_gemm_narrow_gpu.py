"""Narrow tiles for products of few rows: every tile gives the persistent kernels' bits (one chain of MMAs over K), at the
edges of the row boxes and tiles, for a reduction of one k-block and more than the ring holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 512, 512), (16, 520, 64), (17, 1000, 2056), (32, 4096, 520), (33, 4744, 1032),
                                   (64, 9480, 512), (5, 96, 4104), (16, 640, 320), (30, 648, 448), (64, 520, 576)])
def test_bits(M, N, K, b_mn):
    from ferrum_b200 import _lib
    from ferrum_b200.utils import runtime as rt

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, bias = rand(M, K).bfloat16(), rand(N)
    b = rand(K, N).bfloat16() if b_mn else rand(N, K).bfloat16()
    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream

    def run(fn, *tile):
        out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
        _lib.check(fn(a.data_ptr(), b.data_ptr(), out.data_ptr(), None, bias.data_ptr(), M, N, K, K, b.stride(0), N, 0,
                      int(b_mn), 1, 0, 0, *tile, rt.status_ptr(), st), "gemm")
        rt.check_status()
        return out

    want = run(lib.fb_gemm_bf16, 0)
    ref = a.double() @ (b.double() if b_mn else b.double().t()) + bias.double()
    assert (want.double() - ref).norm() <= 2.0 ** -8 * ref.norm()
    tiles = [0, 160, 192, 256] + [t for t in (16, 32, 64) if M <= t]
    for tile in tiles:
        assert torch.equal(run(lib.fb_gemm_bf16_narrow, tile), want), tile
    a[0, K - 1] = float("inf")  # a row's alone
    spoiled = run(lib.fb_gemm_bf16, 0)
    assert not torch.isfinite(spoiled[0]).any() and torch.equal(spoiled[1:], want[1:])
    for tile in tiles:
        assert torch.equal(run(lib.fb_gemm_bf16_narrow, tile).view(torch.int16), spoiled.view(torch.int16)), tile
