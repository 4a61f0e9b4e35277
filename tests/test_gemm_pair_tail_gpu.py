"""The last round of the CTA-pair GEMM in half tiles: with few pairs (the limit on CTAs) small products have one.  The sums are
the single-CTA kernel's, so the bits are the same; the fp64 bound is that of the result's rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [4, 8])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(768, 256, 64), (600, 200, 328), (520, 520, 136), (1304, 136, 520), (512, 1288, 72)])
def test_bits(M, N, K, a_mn, b_mn, ctas):
    from ferrum_b200 import _lib
    from ferrum_b200.utils import runtime as rt

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a = rand(K, M).bfloat16() if a_mn else rand(M, K).bfloat16()
    b = rand(K, N).bfloat16() if b_mn else rand(N, K).bfloat16()
    bias = rand(N)
    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t()) + bias.double()

    def run(fn, limit, dtype, beta, dual):
        out, grad = (torch.ones(M, N, device="cuda", dtype=dtype) for _ in range(2))
        _lib.check(fn(a.data_ptr(), b.data_ptr(), out.data_ptr(), grad.data_ptr() if dual else None, bias.data_ptr(), M, N, K,
                      a.stride(0), b.stride(0), N, int(a_mn), int(b_mn), int(dtype == torch.bfloat16), 2 if dual else 0, beta,
                      limit, rt.status_ptr(), st), "gemm")
        rt.check_status()
        return out, grad

    for dtype, beta, dual in ((torch.bfloat16, 0, False), (torch.bfloat16, 0, True), (torch.float32, 0, False),
                              (torch.float32, 1, False)):
        got, want = run(lib.fb_gemm_bf16_2cta, ctas, dtype, beta, dual), run(lib.fb_gemm_bf16, 0, dtype, beta, dual)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        if not dual:
            tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
            assert (got[0].double() - beta - ref).norm() <= tol * ref.norm()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_tf32(a_mn, b_mn):
    from ferrum_b200 import _lib
    from ferrum_b200.utils import runtime as rt

    M, N, K = 776, 516, 100
    a = torch.randn(*((K, M) if a_mn else (M, K)), device="cuda")
    b = torch.randn(*((K, N) if b_mn else (N, K)), device="cuda")
    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream
    outs = []
    for limit in (8, 0):
        out = torch.empty(M, N, device="cuda")
        _lib.check(lib.fb_gemm_tf32_2cta(a.data_ptr(), b.data_ptr(), out.data_ptr(), None, M, N, K, a.stride(0), b.stride(0), N,
                                         int(a_mn), int(b_mn), 0, 0, limit, rt.status_ptr(), st), "gemm")
        rt.check_status()
        outs.append(out)
    assert torch.equal(*outs)
