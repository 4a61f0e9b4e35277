"""Whole-sequence LSTM / GRU kernels against torch's fp64 recurrence, at the edges of their plans.

Bound: fp32 sums over at most a few hundred terms per step and a contracting recurrence: 2e-5 of each result's norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["LSTM", "GRU"])
@pytest.mark.parametrize("T,B,I,H,L,state", [(1, 1, 3, 8, 1, False), (1, 3, 5, 40, 1, True), (5, 33, 7, 33, 2, True),
                                             (9, 130, 16, 64, 1, False), (4, 37, 12, 257, 1, True),
                                             (3, 150, 8, 512, 1, True), (6, 2, 8, 376, 2, False)])
def test_sequence(kind, T, B, I, H, L, state):
    import ferrum_b200 as fb
    from ferrum_b200 import nn

    torch.manual_seed(T + B + H)
    m = getattr(nn, kind)(I, H, L, device=fb.Device.Cuda(0))
    assert fb.ops.functional.rnn_sequence_ok(4 if kind == "LSTM" else 3, torch.empty(T, B, I, device="cuda"),
                                             m.cells[0].weight_hh)
    ref = getattr(torch.nn, kind)(I, H, L, device="cuda", dtype=torch.float64)
    with torch.no_grad():
        for l, c in enumerate(m.cells):
            for n in ("weight_ih", "weight_hh", "bias_ih", "bias_hh"):
                getattr(ref, f"{n}_l{l}").copy_(getattr(c, n))
    x = torch.randn(T, B, I, device="cuda", requires_grad=True)
    h0 = torch.randn(L, B, H, device="cuda", requires_grad=True) if state else None
    c0 = torch.randn(L, B, H, device="cuda", requires_grad=True) if state and kind == "LSTM" else None
    xd, hd, cd = (t.detach().double().requires_grad_(True) if t is not None else None for t in (x, h0, c0))
    if kind == "LSTM":
        y, (hn, cn) = m.forward_seq(x, (h0, c0) if state else None)
        yr, (hr, cr) = ref(xd, (hd, cd) if state else None)
    else:
        y, hn = m.forward_seq(x, h0)
        yr, hr = ref(xd, hd)
        cn, cr = hn, hr
    g = torch.randn_like(y)
    ((y * g).sum() + (hn * 0.5).sum() + (cn * 0.3).sum()).backward()
    ((yr * g.double()).sum() + (hr * 0.5).sum() + (cr * 0.3).sum()).backward()
    pairs = [(y, yr), (hn, hr), (cn, cr), (x.grad, xd.grad)]
    pairs += [(t.grad, r.grad) for t, r in ((h0, hd), (c0, cd)) if t is not None]
    for l, c in enumerate(m.cells):
        pairs += [(getattr(c, n).grad, getattr(ref, f"{n}_l{l}").grad) for n in
                  ("weight_ih", "weight_hh", "bias_ih", "bias_hh")]
    for got, want in pairs:
        assert (got.double() - want).norm() <= 2e-5 * want.norm() + 1e-6
    with torch.no_grad():
        again = m.forward_seq(x.detach(), None if not state else ((h0, c0) if kind == "LSTM" else h0))[0]
    assert torch.equal(again, y)


@pytest.mark.parametrize("kind", ["LSTM", "GRU"])
@pytest.mark.parametrize("H,bs", [(256, 1), (256, 2), (256, 3), (128, 3), (256, 4), (128, 4), (256, 8)])
def test_batch_slices(kind, H, bs):
    """Every number of batch rows per cluster, the last slice whole and not; how many clusters the chip holds decides which
    batches that are."""
    from ferrum_b200 import _lib

    gates = 4 if kind == "LSTM" else 3
    plans = {B: [_lib.native().rnn_seq_plan(gates, B, H, back) for back in (0, 1)] for B in range(1, 200)}
    sizes = [B for B, p in plans.items() if p[0] % 16 == p[1] % 16 == bs]
    assert sizes, plans
    if bs <= 4:  # weights in registers; for LSTM 256 (four rows of 16 weights per thread in either direction) unrolled
        assert all(p & 16 for B in sizes for p in plans[B])
        assert all(p & 32 for B in sizes for p in plans[B]) or H != 256 or kind != "LSTM"
    whole = max(B for B in sizes if B % bs == 0)
    for B in {whole, whole - 1, sizes[0]} & set(sizes):
        test_sequence(kind, 3, B, 5, H, 1, True)


@pytest.mark.parametrize("kind", ["LSTM", "GRU"])
@pytest.mark.parametrize("how", ["cell_cls", "one_cell", "other_type"])
def test_cells_of_the_users_own(kind, how):
    """A cell class with its own step, in every layer or in one, and a layer of another type than fp32: step by step."""
    import ferrum_b200 as fb
    from ferrum_b200 import nn
    from ferrum_b200.nn import rnn

    calls = []

    class Cell(getattr(rnn, f"{kind}Cell")):
        def step(self, *a):
            calls.append(1)
            return super().step(*a)

    dev = fb.Device.Cuda(0)
    base = getattr(nn, kind)
    torch.manual_seed(4)
    want = base(8, 40, 2, device=dev)
    model = type("Own", (base,), {"cell_cls": Cell})(8, 40, 2, device=dev) if how == "cell_cls" else base(8, 40, 2, device=dev)
    model.load_state_dict(want.state_dict())
    if how == "one_cell":
        model.cells[1].__class__ = Cell
    x = torch.randn(5, 3, 8, device="cuda")
    ref = want.forward_seq(x)[0]
    if how == "other_type":
        with torch.no_grad():
            for n in ("weight_hh", "weight_ih"):
                setattr(model.cells[1], n, torch.nn.Parameter(getattr(model.cells[1], n).to(torch.bfloat16)))
    got = model.forward_seq(x)[0]
    assert len(calls) == {"cell_cls": 10, "one_cell": 5, "other_type": 0}[how]
    assert (got - ref).norm() <= (2e-2 if how == "other_type" else 1e-6) * ref.norm()


@pytest.mark.parametrize("kind", ["LSTM", "GRU"])
@pytest.mark.parametrize("H,B", [(256, 40), (33, 5), (512, 3)])
def test_values_that_are_not_finite(kind, H, B):
    """A NaN stays in its batch row, though rows share a cluster's messages."""
    import ferrum_b200 as fb
    from ferrum_b200 import nn

    torch.manual_seed(H)
    m = getattr(nn, kind)(4, H, 1, device=fb.Device.Cuda(0))
    base, gy = torch.randn(4, B, 4, device="cuda"), torch.randn(4, B, H, device="cuda")

    def run(x):
        x = x.clone().requires_grad_(True)
        y = m.forward_seq(x)[0]
        y.backward(gy)
        return y.detach(), x.grad

    clean = run(base)
    x = base.clone()
    x[1, B // 2] = float("nan")
    others = torch.arange(B, device="cuda") != B // 2
    (y, dx), (yc, dxc) = run(x), clean
    assert torch.equal(y[:, others], yc[:, others]) and torch.equal(dx[:, others], dxc[:, others])
    assert torch.equal(y[0], yc[0]) and torch.isnan(y[1:, B // 2]).all() and torch.isnan(dx[:, B // 2]).all()
