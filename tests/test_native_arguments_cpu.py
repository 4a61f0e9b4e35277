"""Arguments that the native host path refuses before any kernel gets a pointer (sizes and devices; no GPU needed)."""
import pytest
import torch


def _native():
    from ferrum_b200 import _lib

    return _lib.native()


@pytest.mark.parametrize("gates", [3, 4])
@pytest.mark.parametrize("state,what", [((2, 8), "initial state"), ((1, 8), "initial state"), ((3, 9), "initial state"),
                                        ((8,), "initial state"), ("meta", "on meta")])
def test_initial_states(gates, state, what):
    """An input of batch 3, hidden size 8: other sizes and devices of the hidden or the cell state."""
    proj, w = torch.zeros(2, 3, gates * 8), torch.zeros(gates * 8, 8)
    bad = torch.zeros(3, 8, device="meta") if state == "meta" else torch.zeros(*state)
    with pytest.raises(ValueError, match=what):
        _native().rnn_seq(gates, proj, w, None, bad, None)
    with pytest.raises(ValueError, match=what):
        _native().rnn_seq(gates, proj, w, None, None, bad)


def test_recurrent_matrix_and_bias():
    proj, w = torch.zeros(2, 3, 32), torch.zeros(32, 8)
    for args in ((proj, torch.zeros(32, 7), None), (proj[0], w, None), (proj, w, torch.zeros(31)),
                 (proj, w.to("meta"), None), (proj, w, torch.zeros(32, device="meta")), (proj, w, None)):
        with pytest.raises(ValueError):
            _native().rnn_seq(4, *args, None, None)


def test_nll_targets():
    lp = torch.zeros(4, 5)
    for bad in (torch.zeros(3, dtype=torch.int64), torch.zeros(5, dtype=torch.int64)):
        with pytest.raises(ValueError, match="one target per row"):
            _native().nll(lp, bad)
    with pytest.raises(ValueError, match="on meta"):
        _native().nll(lp, torch.zeros(4, dtype=torch.int64, device="meta"))
    with pytest.raises(ValueError, match="one target per row"):
        _native().nll(lp[:0], torch.zeros(0, dtype=torch.int64))


def test_cross_entropy_labels():
    x = torch.zeros(4, 5)
    for n in (3, 5):
        with pytest.raises(ValueError, match="one label per row"):
            _native().cross_entropy(x, torch.zeros(n, dtype=torch.int64))
    with pytest.raises(ValueError, match="on meta"):
        _native().cross_entropy(x, torch.zeros(4, dtype=torch.int64, device="meta"))


def test_elementwise_targets_and_embedding_indices():
    x, i = torch.zeros(4, 5), torch.zeros(2, 3, dtype=torch.int64)
    for bad in (torch.zeros(4, 4), torch.zeros(20), torch.zeros(4, 5, device="meta")):
        with pytest.raises(ValueError):
            _native().elementwise_loss(x, bad, 0)
    for weight, idx, pool in ((x, i.to("meta"), False), (x, i.to("meta"), True), (x, i[0], True), (x[0], i, False)):
        with pytest.raises(ValueError):
            _native().embedding(weight, idx, -1, pool, False, None)


@pytest.mark.parametrize("shape", [(0, 5), (4, 0), (0, 0)])
def test_no_mean_over_nothing(shape):
    """The native op refuses, and so do the C entry points, which return before they touch their pointers."""
    from ferrum_b200 import _lib

    with pytest.raises(ValueError, match="empty"):
        _native().cross_entropy(torch.zeros(shape), torch.zeros(shape[0], dtype=torch.int64))
    lib = _lib.cuda()
    assert lib.fb_ce_fwd(None, None, None, None, None, *shape, 1.0, 0, None) != 0
    assert lib.fb_nll_fwd(None, None, None, None, *shape, 1.0, 0, None, None) != 0
    assert lib.fb_loss_mean_fwd(None, None, None, None, 0, 0, 1.0, None) != 0


def test_products_that_no_kernel_has():
    """Mixed operand types, fp32 operands with a bf16 result, accumulation onto a bf16 result, an unknown activation."""
    f, h = torch.zeros(8, 8), torch.zeros(8, 8, dtype=torch.bfloat16)
    for a, b, out, act, acc in ((f, h, f, 0, False), (h, f, f, 0, False), (f, f, h, 0, False), (h, h, h, 0, True),
                                (f, f, f, 6, False)):
        with pytest.raises(RuntimeError, match="gemm"):
            _native().gemm_nt(a, b, None, act, out, acc, False)


def test_biases_and_scales():
    """A bias or a scale on another device than the weight, or of another size, in the three ops that read one by a pointer."""
    x, w, ok = torch.zeros(4, 6), torch.zeros(5, 6), torch.zeros(5)
    for bad, what in ((torch.zeros(5, device="meta"), "on meta"), (torch.zeros(4), "expected 5"), (torch.zeros(6), "expected 5")):
        with pytest.raises(ValueError, match=what):
            _native().linear(x, w, bad, 0, False, False, None, None)
        for args in ((bad, ok, ok), (ok, bad, ok), (ok, ok, bad)):
            with pytest.raises(ValueError, match=what):
                _native().linear_act_norm(x, w, *args, 1e-5, 0, False, False, None, None)
        for args in ((bad, ok), (ok, bad), (None, bad)):
            with pytest.raises(ValueError, match=what):
                _native().layer_norm(torch.zeros(4, 5), *args, 1e-5, 0)
