"""Rows of any pitch and address copied to an aligned pitch: every misalignment, widths around a 16-byte piece, the last
words of a matrix; and results of odd pitch from the CTA-pair kernel.  Copies are exact."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 7, 8, 9, 15, 17, 64, 333, 1001])
@pytest.mark.parametrize("rows,extra", [(1, 0), (5, 0), (37, 3), (300, 8)])
def test_copies(rows, cols, extra):
    from ferrum_b200 import _lib

    lib, st, to = _lib.cuda(), torch.cuda.current_stream().cuda_stream, -(-cols // 8) * 8
    pitch = cols + extra
    for off in range(8):
        # any 16 bits, NaNs among them
        flat = torch.randint(-2 ** 15, 2 ** 15, (off + rows * pitch,), device="cuda", dtype=torch.int16)
        src = flat[off:].view(rows, pitch)[:, :cols]
        out = [torch.full((rows, to), 3, device="cuda", dtype=torch.int16) for _ in range(2)]
        half = (rows + 1) // 2
        _lib.check(lib.fb_repack_rows(src.data_ptr(), out[0].data_ptr(), rows, cols, pitch, src.data_ptr(),
                                      out[1].data_ptr(), half, cols, pitch, st), "fb_repack_rows")
        assert torch.equal(out[0][:, :cols], src) and not out[0][:, cols:].any()
        assert torch.equal(out[1][:half, :cols], src[:half]) and (out[1][half:] == 3).all()


@pytest.mark.parametrize("M,N,K", [(512, 129, 64), (513, 257, 128), (1000, 1001, 72), (2047, 255, 512)])
def test_results_of_odd_pitch(M, N, K):
    """fp32 sums: 2^-23 per 16 of K (the tensor core truncates); bf16: 2^-9; a value beside its derivative."""
    from ferrum_b200.ops import gemm
    from ferrum_b200.utils.runtime import check_status

    a, b = (torch.randn(n, K, device="cuda").bfloat16() for n in (M, N))
    ref = a.double() @ b.double().t()
    out = torch.full((M, N), 2.0, device="cuda")
    gemm.gemm_bf16(a, b, out=out, accumulate=True)
    assert (out.double() - 2 - ref).norm() <= (K / 16 * 2.0 ** -23 + 1e-6) * (ref.norm() + 2 * (M * N) ** 0.5)
    low, der = (torch.full((M, N), 3.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    gemm.gemm_bf16(a, b, act="relu", out=low, act_grad=der)
    check_status()
    assert (low.double() - ref.clamp_min(0)).norm() <= 2.0 ** -8 * ref.norm()
    sure = ref.abs() > 1e-3
    assert torch.equal(der[sure] > 0, ref[sure] > 0) and ((der == 0) | (der == 1)).all()
