"""Chains of few-row products and normalisations, whose kernels start beside the tail of the one ahead: the results are
those of the same chain with a synchronisation after every kernel, with buffers reused at once and under capture."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other", [True, False])
@pytest.mark.parametrize("rows,width,deep", [(16, 4096, 6), (1, 1024, 5), (64, 2048, 4), (33, 1032, 3)])
def test_chain(rows, width, deep, other):
    """``other``: a kernel that is nobody's dependent between the layers; without it every one waits for the one ahead,
    which itself may still be waiting."""
    from ferrum_b200.ops import functional as F
    from ferrum_b200.ops import gemm  # noqa: F401
    from ferrum_b200 import _lib
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(width)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    ws = [(rand(width, width) * width ** -0.5).bfloat16() for _ in range(deep)]
    gamma, beta = rand(width), rand(width)

    def chain(x, sync=False):
        for w in ws:
            y = torch.empty(rows, width, device="cuda", dtype=torch.bfloat16)
            _lib.native().gemm_nt(x, w, None, 0, y, False, False)
            if sync:
                torch.cuda.synchronize()
            x = F.layer_norm(y, gamma, beta)
            if sync:
                torch.cuda.synchronize()
            if other:
                w.mul_(1.0)  # the next product's weights may have been written just now
        return x

    with torch.no_grad():
        xs = [rand(rows, width).bfloat16() for _ in range(8)]
        want = [chain(x, True) for x in xs]
        for _ in range(3):
            assert all(torch.equal(chain(x), w) for x, w in zip(xs, want))
        static = xs[0].clone()
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            chain(static)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                out = chain(static)
        torch.cuda.current_stream().wait_stream(s)
        for x, w in zip(xs, want):
            static.copy_(x)
            graph.replay()
            assert torch.equal(out, w)
    check_status()
