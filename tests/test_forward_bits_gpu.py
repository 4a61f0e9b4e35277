"""A bf16 forward pass over aligned rows has one order of summation: neither the recording of gradients, nor the rows that
share a batch, nor the kernel that a number of rows selects changes a bit, at sizes where weight gradients divide their
reduction."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,din,dout", [(1, 2048, 130), (1, 512, 512), (16, 4096, 4096), (17, 520, 1001), (32, 1000, 4096),
                                           (33, 4096, 1000), (64, 2048, 513), (65, 2048, 512), (96, 4096, 1000),
                                           (300, 8192, 512)])
def test_no_grad_and_row_subsets(rows, din, dout):
    import ferrum_b200 as fb
    from ferrum_b200 import nn
    from ferrum_b200.ops.gemm import gemm_bf16

    torch.manual_seed(rows)
    lin = nn.Linear(din, dout, device=fb.Device.Cuda(0))
    x = torch.randn(rows, din, device="cuda").bfloat16()
    with fb.autocast():
        trained = lin(x).detach()
        with fb.no_grad():
            assert torch.equal(lin(x), trained)
            assert torch.equal(lin(x[: (rows + 1) // 2].contiguous()), trained[: (rows + 1) // 2])
    assert torch.equal(gemm_bf16(x, lin.weight.detach().bfloat16(), bias=lin.bias.detach()), trained)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("tile,M,N,K", [(16, 1, 512, 512), (16, 16, 1000, 520), (32, 17, 513, 1000), (32, 32, 640, 576),
                                        (192, 33, 1001, 512), (192, 64, 575, 4103)])
def test_narrow_tiles_are_the_persistent_kernels(tile, M, N, K, a_mn, b_mn):
    """Bit for bit, with every epilogue."""
    from ferrum_b200 import _lib
    from ferrum_b200.ops.gemm import ACT, _major, gemm_bf16
    from ferrum_b200.utils import runtime as rt

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    pad = lambda n: -(-n // 8) * 8

    def operand(rows, mn):
        if mn:
            return torch.randn(K, pad(rows), device="cuda", generator=g).bfloat16()[:, :rows].t()
        return torch.randn(rows, pad(K), device="cuda", generator=g).bfloat16()[:, :K]

    a, b, bias = operand(M, a_mn), operand(N, b_mn), torch.randn(N, device="cuda", generator=g)

    def both(act, out_dtype, accumulate, act_grad):
        res = []
        for narrow in (False, True):
            out = torch.full((M, N + 3), 2.0, device="cuda", dtype=out_dtype)[:, :N]
            der = torch.empty(M, N + 3, device="cuda", dtype=out_dtype)[:, :N] if act_grad else None
            if narrow:
                (am, lda), (bm, ldb) = _major(a), _major(b)
                _lib.check(_lib.cuda().fb_gemm_bf16_narrow(
                    a.data_ptr(), b.data_ptr(), out.data_ptr(), None if der is None else der.data_ptr(), bias.data_ptr(),
                    M, N, K, lda, ldb, out.stride(0), am, bm, int(out_dtype == torch.bfloat16), ACT[act], accumulate,
                    tile, rt.status_ptr(), torch.cuda.current_stream().cuda_stream), "fb_gemm_bf16_narrow")
            else:
                gemm_bf16(a, b, bias=bias, act=act, out=out, accumulate=bool(accumulate), act_grad=der)
            res.append((out, der))
        rt.check_status()
        assert torch.equal(res[0][0], res[1][0]) and (der is None or torch.equal(res[0][1], res[1][1]))

    for act in ACT:
        both(act, torch.bfloat16, 0, False)
    both("gelu", torch.bfloat16, 0, True)
    both(None, torch.float32, 1, False)
