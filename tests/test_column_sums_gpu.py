"""Column sums of a matrix against fp64, in one launch of clusters or added up in a cleared buffer: alone and behind the gradient
of an activation; and the column statistics of the LayerNorm backward, whose kernel clears what its fold adds to.  Bound: an
addition errs by at most 2^-24 of the partial sum; those of normal numbers of both signs stay below a sixteenth of the summed
magnitudes once there are many, so 2^-19 of these covers some five hundred additions in a row (a thread's, a warp's, the
blocks'); bf16 values are summed as they are stored."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 4096), (63, 7), (64, 8), (65, 33), (128, 256), (511, 1000), (513, 1184), (777, 37), (1025, 1001), (4096, 2048),
          (70000, 3), (20000, 64), (16384, 1024), (8193, 1001)]


def _bound(x):
    return 2.0 ** -19 * x.double().abs().sum(0) + 1e-30


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", SHAPES)
def test_sums(rows, cols, dtype):
    from ferrum_b200 import _lib
    from ferrum_b200.ops import functional as F

    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    for off in (0, 1):  # behind a 16-byte boundary: one by one
        x = torch.randn(rows * cols + 1, device="cuda", generator=g).to(dtype)[off:][:rows * cols].view(rows, cols)
        out = torch.full((cols,), float("nan"), device="cuda")
        F.raw_colsum(x, out)
        assert ((out - x.double().sum(0)).abs() <= _bound(x)).all()
        F.raw_colsum(x, out, accumulate=True)
        assert ((out - 2 * x.double().sum(0)).abs() <= 3 * _bound(x)).all()
        if _lib.cuda().fb_colsum_clusters(rows, cols, F._dt(x), 0, off == 0):  # no atomics: the same bits again
            assert torch.equal(F.raw_colsum(x), F.raw_colsum(x))


@pytest.mark.parametrize("act", [1, 4, 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", SHAPES[:-4])
def test_behind_an_activation(rows, cols, dtype, act):
    from ferrum_b200 import _lib
    from ferrum_b200.ops import functional as F

    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    dt = F._dt(torch.empty(0, dtype=dtype))
    for off in (0, 1):
        dy, y, d, want = (torch.randn(rows * cols + 1, device="cuda", generator=g).to(dtype)[off:][:rows * cols].view(rows, cols)
                          for _ in range(4))
        sums = torch.full((cols,), float("nan"), device="cuda")
        d.fill_(float("nan"))
        _lib.check(lib.fb_unary_bwd(dy.data_ptr(), y.data_ptr(), want.data_ptr(), rows * cols, act, 0.0, 0.0, dt, st), "two")
        rc = lib.fb_unary_bwd_colsum(dy.data_ptr(), y.data_ptr(), d.data_ptr(), sums.data_ptr(), rows, cols, act, dt, st)
        if lib.fb_colsum_clusters(rows, cols, dt, 1, off == 0):
            assert rc == 0 and torch.equal(d, want)
            assert ((sums - d.double().sum(0)).abs() <= _bound(d)).all()
        else:
            assert rc == -3 and d.isnan().all() and sums.isnan().all()
    assert lib.fb_unary_bwd_colsum(dy.data_ptr(), y.data_ptr(), d.data_ptr(), sums.data_ptr(), rows, cols, 3, dt, st) == -1


@pytest.mark.parametrize("rows,cols,size,grad,aligned,one", [
    (128, 256, 2, 1, True, True), (1024, 4096, 2, 1, True, True), (8192, 4096, 2, 1, True, True), (8192, 4096, 4, 1, True, True),
    # elements one by one: a round of the block's threads behind a gradient
    (512, 1001, 2, 1, True, True), (513, 1001, 2, 1, True, False), (512, 1001, 4, 1, True, True), (1025, 1001, 4, 1, True, False),
    (8191, 4095, 2, 1, True, False), (8191, 4095, 4, 1, True, False), (64, 1024, 2, 1, False, True), (8192, 1024, 2, 1, False, False),
    # a few for sums alone: a bias of few outputs over many rows
    (4096, 1, 2, 0, True, True), (4097, 1, 2, 0, True, False), (16384, 1, 4, 0, True, True), (16385, 1, 4, 0, True, False),
    (1 << 20, 1, 4, 0, True, False), (32768, 1001, 4, 0, True, True), (32776, 1001, 4, 0, True, False), (8192, 1001, 2, 0, True, False),
    # whole pieces: 96 KB to a block, or wide ranges
    (24576, 64, 2, 1, True, True), (24608, 64, 2, 1, True, False), (32768, 64, 2, 0, True, True), (32776, 64, 2, 0, True, False),
    (131072, 8, 4, 0, True, True), (131072, 8, 4, 1, True, False), (32768, 160, 4, 1, True, False), (32768, 1024, 4, 0, True, True),
    (32768, 512, 2, 1, True, False), (32768, 512, 4, 1, True, True), (16384, 1024, 2, 0, True, False),
    (8192, 2048, 2, 0, True, True), (8200, 2048, 2, 0, True, False),
])
def test_which_launches(rows, cols, size, grad, aligned, one):
    from ferrum_b200 import _lib

    assert bool(_lib.cuda().fb_colsum_clusters(rows, cols, 3 if size == 2 else 0, grad, aligned)) == one


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
@pytest.mark.parametrize("rows,width", [(512, 1001), (1025, 1001), (300, 4095), (1025, 1024)])
def test_bias_gradient_of_a_linear_layer_with_relu(rows, width, prec):
    """Either way in a backward pass: the bias' gradient is the column sum of the gradient behind the ReLU."""
    import contextlib

    import ferrum_b200 as fb
    from ferrum_b200.ops import functional as F

    g = torch.Generator(device="cuda").manual_seed(rows)
    x, w = (torch.randn(n, 24, device="cuda", generator=g) for n in (rows, width))
    b = torch.zeros(width, device="cuda", requires_grad=True)
    with fb.autocast() if prec == "bf16" else contextlib.nullcontext():
        y = F.linear(x, w, b, act="relu")
    gy = torch.randn(y.shape, device="cuda", generator=g).to(y.dtype)
    y.backward(gy)
    d = gy * (y > 0)
    assert ((b.grad - d.double().sum(0)).abs() <= _bound(d)).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 1001), (40, 96), (300, 1024), (777, 1001), (2049, 4096), (5, 9000)])
def test_layernorm_statistics_are_written_or_added(rows, cols, dtype):
    from ferrum_b200 import _lib
    from ferrum_b200.ops import functional as F
    from ferrum_b200.utils.runtime import check_status

    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, dy = (torch.randn(rows, cols, device="cuda", generator=g).to(dtype) for _ in range(2))
    gamma = torch.ones(cols, device="cuda")
    mean, rstd = x.float().mean(1), (x.float().var(1, unbiased=False) + 1e-5).rsqrt()
    dx, nblk = torch.empty_like(x), lib.fb_layernorm_bwd_blocks(rows, cols)
    partial = torch.empty(max(nblk, 1), 3, cols, device="cuda")
    ones, nan = torch.ones(3, cols, device="cuda"), torch.full((3, cols), float("nan"), device="cuda")
    for stats, flags in ((ones, 1), (nan, 3)):
        _lib.check(lib.fb_layernorm_bwd(dy.data_ptr(), x.data_ptr(), None, gamma.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
                                        dx.data_ptr(), partial.data_ptr(), stats.data_ptr(), rows, cols, 0,
                                        F._dt(x), nblk, flags, st), "ln")
    check_status()
    xh = (x.double() - mean.double()[:, None]) * rstd.double()[:, None]
    terms = torch.stack([dy.double() * xh, dy.double(), dx.double()])
    size = terms.abs().sum(1)
    # the column sum of dx is that of the values before they are rounded to the type
    tol = 2.0 ** -18 * size + torch.tensor([0.0, 0.0, 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20], device="cuda")[:, None] * size
    assert ((nan - terms.sum(1)).abs() <= tol + 1e-6).all() and ((ones - 1 - terms.sum(1)).abs() <= tol + 1e-5).all()
