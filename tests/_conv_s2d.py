"""The space-to-depth form of a strided convolution in plain torch, as csrc/kernels/conv_layout.cu lays it out: with
``z[b, I, J, (rh, rw, c)] = x[b, c, I * sh + rh - ph, J * sw + rw - pw]``, rh < min(sh, kh), rw < min(sw, kw), a convolution
of stride (sh, sw) with a kh x kw filter is one of stride 1 with a ceil(kh / sh) x ceil(kw / sw) filter."""
import torch


def geometry(x_shape, w_shape, stride, padding):
    """Ho, Wo, k2h, k2w, Hz, Wz, eh, ew, channels of z (padded to 8)."""
    B, C, H, W = x_shape
    O, _, kh, kw = w_shape
    (sh, sw), (ph, pw) = stride, padding
    Ho, Wo = (H + 2 * ph - kh) // sh + 1, (W + 2 * pw - kw) // sw + 1
    k2h, k2w, eh, ew = -(-kh // sh), -(-kw // sw), min(sh, kh), min(sw, kw)
    return Ho, Wo, k2h, k2w, Ho + k2h - 1, Wo + k2w - 1, eh, ew, -(-eh * ew * C // 8) * 8


def pack_input(x, w_shape, stride, padding):
    """x [B, C, H, W] -> z [B, Hz, Wz, Cz]."""
    B, C, H, W = x.shape
    (sh, sw), (ph, pw) = stride, padding
    _, _, _, _, Hz, Wz, eh, ew, Cz = geometry(x.shape, w_shape, stride, padding)
    xp = torch.nn.functional.pad(x, (pw, Wz * sw, ph, Hz * sh))[:, :, :Hz * sh, :Wz * sw]  # zero outside the image
    z = xp.reshape(B, C, Hz, sh, Wz, sw)[:, :, :, :eh, :, :ew].permute(0, 2, 4, 3, 5, 1).reshape(B, Hz, Wz, eh * ew * C)
    return torch.nn.functional.pad(z, (0, Cz - eh * ew * C))


def pack_filters(w, stride, pitch):
    """w [O, C, kh, kw] -> [O, k2h * k2w, pitch]; taps that do not exist are zero."""
    O, C, kh, kw = w.shape
    sh, sw = stride
    k2h, k2w, eh, ew = -(-kh // sh), -(-kw // sw), min(sh, kh), min(sw, kw)
    out = w.new_zeros(O, C, k2h * sh, k2w * sw)
    out[:, :, :kh, :kw] = w
    out = out.view(O, C, k2h, sh, k2w, sw)[:, :, :, :eh, :, :ew].permute(0, 2, 4, 3, 5, 1).reshape(O, k2h * k2w, eh * ew * C)
    return torch.nn.functional.pad(out, (0, pitch - eh * ew * C))


SHAPES = [(2, 3, 5, 17, 19, (3, 3), (2, 2), (1, 1)), (1, 4, 6, 16, 16, (4, 4), (4, 4), (0, 0)),
          (2, 5, 7, 15, 20, (5, 3), (2, 3), (2, 1)), (1, 3, 4, 14, 14, (7, 7), (2, 2), (3, 3)),
          (2, 16, 9, 12, 13, (1, 1), (2, 2), (0, 0)), (1, 65, 8, 11, 9, (1, 3), (3, 2), (0, 1)),
          (2, 72, 3, 10, 70, (3, 3), (1, 1), (0, 0)), (1, 130, 64, 9, 8, (2, 2), (2, 1), (0, 0))]
