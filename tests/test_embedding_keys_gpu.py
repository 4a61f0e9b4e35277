"""Sorted scatter of embedding gradients behind 32-bit keys: indices outside the table, padding, one row, repeats; an fp64
sum is the oracle (2^-22 of the summed magnitudes for up to a few hundred fp32 additions per row)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab,n,dim", [(1, 1, 4), (1, 300, 7), (5, 33, 64), (1000, 4097, 12), (70000, 511, 8)])
@pytest.mark.parametrize("padding", [-1, 0])
def test_gradient(vocab, n, dim, padding):
    from ferrum_b200 import _lib
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(vocab + n)
    idx = torch.randint(0, vocab, (n,), device="cuda", generator=g)
    bad = idx.clone()
    bad[::5] = torch.tensor([vocab, -1, 2 ** 40, -2 ** 40], device="cuda").repeat(n)[: bad[::5].numel()]
    dout = torch.randn(n, dim, device="cuda", generator=g)
    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream
    for ids in (idx, bad):
        keys, rows = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
        _lib.check(lib.fb_embedding_pairs(ids.data_ptr(), keys.data_ptr(), rows.data_ptr(), n, vocab, 1, st), "fb_embedding_pairs")
        ok = (ids >= 0) & (ids < vocab)
        assert torch.equal(keys.long(), torch.where(ok, ids, vocab))
        ok_grad = ok & (ids != padding)
        want, size = (torch.zeros(vocab, dim, device="cuda", dtype=torch.float64) for _ in range(2))
        want.index_add_(0, ids[ok_grad], dout[ok_grad].double())
        size.index_add_(0, ids[ok_grad], dout[ok_grad].double().abs())
        for unsorted in (keys, torch.where(ok, ids, vocab)):  # 64 bits: tables of 2^31 - 1 rows and more
            key, perm = torch.sort(unsorted, stable=True)
            dw = torch.zeros(vocab, dim, device="cuda")
            pairs = key.dtype == torch.int32
            scatter, at = (lib.fb_embedding_bwd_pairs, rows[perm]) if pairs else (lib.fb_embedding_bwd_sorted, perm)
            _lib.check(scatter(dout.data_ptr(), key.data_ptr(), at.data_ptr(), dw.data_ptr(), n, dim, 1, 1.0, padding, vocab, 0,
                               st), "scatter")
            check_status()
            assert ((dw - want).abs() <= 2.0 ** -22 * size * 8).all()


@pytest.mark.parametrize("vocab,batch,seq,dim", [(1, 3, 5, 4), (2, 1, 1, 8), (255, 7, 33, 12), (256, 64, 70, 8), (65536, 9, 31, 5)])
def test_pairs(vocab, batch, seq, dim):
    """Pairs sorted by no more bits than a row number has, index vocab (outside) included; mean of `seq` rows, padding."""
    from ferrum_b200 import _lib
    from ferrum_b200.ops import functional as F
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(vocab)
    n, idx = batch * seq, torch.randint(0, vocab, (batch, seq), device="cuda", generator=g)
    idx.view(-1)[0] = vocab - 1
    lib, st = _lib.cuda(), torch.cuda.current_stream().cuda_stream
    odd = idx.clone().view(-1)
    odd[-1] = vocab + 7
    keys, rows = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    _lib.check(lib.fb_embedding_pairs(odd.data_ptr(), keys.data_ptr(), rows.data_ptr(), n, vocab, seq, st), "pairs")
    assert torch.equal(keys.long(), odd.clamp(max=vocab)) and torch.equal(rows.long(), torch.arange(n, device="cuda") // seq)
    key, perm = torch.sort(keys, stable=True)
    dout, dw = torch.randn(batch, dim, device="cuda", generator=g), torch.zeros(vocab, dim, device="cuda")
    _lib.check(lib.fb_embedding_bwd_pairs(dout.data_ptr(), key.data_ptr(), rows[perm].data_ptr(), dw.data_ptr(), n, dim, seq,
                                          1.0 / seq, -1, vocab, 0, st), "bwd")
    check_status()
    per = dout.double().repeat_interleave(seq, 0) / seq
    want, size = (torch.zeros(vocab, dim, device="cuda", dtype=torch.float64) for _ in range(2))
    want.index_add_(0, odd[:-1], per[:-1])
    size.index_add_(0, odd[:-1], per[:-1].abs())
    assert ((dw - want).abs() <= 2.0 ** -22 * size * 8).all()
    for pool, padding in ((True, None), (False, 0)):
        w = torch.randn(vocab, dim, device="cuda", generator=g).requires_grad_(True)
        y = F.embedding_mean_pool(w, idx) if pool else F.embedding(w, idx, padding_idx=padding)
        gy = torch.randn(y.shape, device="cuda", generator=g)
        y.backward(gy)
        per = (gy.double() / seq).repeat_interleave(seq, 0) if pool else gy.double().reshape(n, dim)
        want, size = (torch.zeros(vocab, dim, device="cuda", dtype=torch.float64) for _ in range(2))
        keep = torch.ones(n, dtype=torch.bool, device="cuda") if padding is None else idx.view(-1) != padding
        want.index_add_(0, idx.view(-1)[keep], per[keep])
        size.index_add_(0, idx.view(-1)[keep], per[keep].abs())
        check_status()
        assert ((w.grad - want).abs() <= 2.0 ** -22 * size * 8).all()


@pytest.mark.parametrize("dim", [3, 8, 36, 1024, 1100])
@pytest.mark.parametrize("vocab,n", [(1, 1), (1, 64), (15, 31), (17, 32), (40, 33), (40, 4000), (3000, 700), (33, 95), (5, 1000)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gradient_in_chunks(vocab, n, dim, dtype):
    """Into a table of zeros and onto another: runs of an index within a chunk of 32, over its edges and over many chunks,
    the same row of the gradient several times in a run, an index that is the padding, indices outside the table.  Sums of
    32 bits within a chunk, then of the chunks, then the table's value."""
    from ferrum_b200 import _lib
    from ferrum_b200.ops import functional as F
    from ferrum_b200.utils.runtime import check_status

    g = torch.Generator(device="cuda").manual_seed(vocab + n + dim)
    keys = torch.randint(0, vocab, (n,), device="cuda", generator=g)
    keys[: n // 2] = vocab // 2
    keys[-1] = vocab
    for padding, zeroed in ((-1, True), (-1, False), (vocab // 2, True)):
        group = 3
        rows = torch.arange(n, device="cuda") // group
        key, perm = torch.sort(keys, stable=True)
        key, row = key.int(), rows[perm].int()
        dout = torch.randn((n + group - 1) // group, dim, device="cuda", generator=g).to(dtype)
        old = torch.randn(vocab, dim, device="cuda", generator=g) * (0 if zeroed else 1)
        dw, lib = old.clone(), _lib.cuda()
        _lib.check((lib.fb_embedding_bwd_pairs_zeroed if zeroed else lib.fb_embedding_bwd_pairs)(
            dout.data_ptr(), key.data_ptr(), row.data_ptr(), dw.data_ptr(), n, dim, group, 0.5, padding, vocab,
            F._dt(dout), torch.cuda.current_stream().cuda_stream), "grad")
        check_status()
        want, size = (torch.zeros(vocab + 1, dim, device="cuda", dtype=torch.float64) for _ in range(2))
        want.index_add_(0, keys, dout.double()[rows] * 0.5)
        size.index_add_(0, keys, dout.double()[rows].abs() * 0.5)
        if padding >= 0:
            want[padding] = 0
        bound = 2.0 ** -24 * (40 + n / 32) * (size[:vocab] + old.abs())
        assert ((dw - old.double() - want[:vocab]).abs() <= bound).all()
