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
        keys = torch.empty(n, dtype=torch.int32, device="cuda")
        _lib.check(lib.fb_embedding_keys(ids.data_ptr(), keys.data_ptr(), n, vocab, st), "fb_embedding_keys")
        ok = (ids >= 0) & (ids < vocab)
        assert torch.equal(keys.long(), torch.where(ok, ids, vocab))
        ok_grad = ok & (ids != padding)
        want, size = (torch.zeros(vocab, dim, device="cuda", dtype=torch.float64) for _ in range(2))
        want.index_add_(0, ids[ok_grad], dout[ok_grad].double())
        size.index_add_(0, ids[ok_grad], dout[ok_grad].double().abs())
        for unsorted in (keys, torch.where(ok, ids, vocab)):  # 64 bits: tables of 2^31 - 1 rows and more
            key, perm = torch.sort(unsorted, stable=True)
            dw = torch.zeros(vocab, dim, device="cuda")
            _lib.check(lib.fb_embedding_bwd_sorted(dout.data_ptr(), key.data_ptr(), key.element_size(), perm.data_ptr(),
                                                   dw.data_ptr(), n, dim, 1, 1.0, padding, vocab, 0, st),
                       "fb_embedding_bwd_sorted")
            check_status()
            assert ((dw - want).abs() <= 2.0 ** -22 * size * 8).all()
