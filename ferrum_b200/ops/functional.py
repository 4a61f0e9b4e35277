"""Differentiable ops on ``torch.Tensor`` values.

Every function here takes and returns plain torch tensors.  For CUDA tensors
(fp32 / bf16) the forward and the backward both run this package's sm_100a
kernels through autograd nodes (most of them native, ``csrc/native``); for CPU tensors the
same mathematics is expressed with torch CPU ops so that the torch autograd
engine differentiates it.  There is no second GPU implementation: if the
native library is missing on a GPU machine the launchers raise.

Formulas follow the reference where it is sound (GELU tanh constants of
ferrum-nn/src/activation.rs:254-262, BCE epsilon of ferrum-nn/src/loss.rs:51-71,
mean over B*C in cross_entropy_loss, loss.rs:119-123) and are mathematically
correct where the reference's tape is not (per-row softmax / LayerNorm,
gradients through scalar ops, embedding backward).
"""
from __future__ import annotations

import math

import torch
from torch.autograd import Function

from .. import _lib, config
from ..utils import runtime as _rt
from . import gemm as _gemm

F32, BF16 = 0, 3

UNARY = {
    "none": 0, "relu": 1, "gelu": 2, "silu": 3, "tanh": 4, "sigmoid": 5, "leaky_relu": 6, "elu": 7, "neg": 8,
    "exp": 9, "log": 10, "sqrt": 11, "abs": 12, "sin": 13, "cos": 14, "pow": 15, "add_scalar": 16,
    "mul_scalar": 17, "rsub_scalar": 18, "rdiv_scalar": 19, "affine": 20, "clamp": 21,
}
BINARY = {"add": 0, "sub": 1, "mul": 2, "div": 3, "pow": 4, "max": 5, "min": 6}
REDUCE = {"sum": 0, "mean": 1, "max": 2, "min": 3, "prod": 4}
LOSS = {"mse": 0, "bce": 1, "l1": 2, "smooth_l1": 3}

GELU_C = 0.7978845608028654
GELU_A = 0.044715


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _dt(t: torch.Tensor) -> int:
    if t.dtype == torch.float32:
        return F32
    if t.dtype == torch.bfloat16:
        return BF16
    raise TypeError(f"kernel supports fp32 / bf16, got {t.dtype}")


def _native(t: torch.Tensor) -> bool:
    """True when `t` is handled by this package's CUDA kernels."""
    return t.is_cuda and t.dtype in (torch.float32, torch.bfloat16)


def _ptr(t):
    return None if t is None else t.data_ptr()


# =============================================================================== raw launchers
def raw_cast(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    if x.dtype == dtype:
        return x
    if x.is_cuda and {x.dtype, dtype} == {torch.float32, torch.bfloat16}:
        x = x.contiguous()
        out = torch.empty_like(x, dtype=dtype)
        _lib.check(_lib.cuda().fb_cast(x.data_ptr(), out.data_ptr(), x.numel(), _dt(x), _dt(out), _stream()),
                   "fb_cast")
        return out
    return x.to(dtype)


def low_copy(x: torch.Tensor) -> torch.Tensor:
    """bf16 copy of a CUDA tensor that needs no gradient, outside the graph; a dual tensor is refused."""
    return _lib.native().low_copy(x)


def raw_unary(x: torch.Tensor, op: str, alpha: float = 0.0, beta: float = 0.0) -> torch.Tensor:
    x = x.contiguous()
    y = torch.empty_like(x)
    _lib.check(_lib.cuda().fb_unary_fwd(x.data_ptr(), y.data_ptr(), x.numel(), UNARY[op], alpha, beta, _dt(x),
                                        _stream()), "fb_unary_fwd")
    return y


def raw_unary_bwd(dy: torch.Tensor, saved, op: str, alpha: float = 0.0, beta: float = 0.0) -> torch.Tensor:
    dy = dy.contiguous()
    if saved is not None:
        saved = saved.contiguous()
        if saved.dtype != dy.dtype:
            saved = raw_cast(saved, dy.dtype)
    dx = torch.empty_like(dy)
    _lib.check(_lib.cuda().fb_unary_bwd(dy.data_ptr(), _ptr(saved), dx.data_ptr(), dy.numel(), UNARY[op], alpha,
                                        beta, _dt(dy), _stream()), "fb_unary_bwd")
    return dx


def raw_binary(a: torch.Tensor, b: torch.Tensor, op: str) -> torch.Tensor:
    """Broadcasting fp32 binary op; operands may be strided / expanded views."""
    import ctypes

    shape = torch.broadcast_shapes(a.shape, b.shape)
    if len(shape) > 6:
        a, b = a.expand(shape).reshape(-1), b.expand(shape).reshape(-1)
        shape = a.shape
    ae, be = a.expand(shape), b.expand(shape)
    out = torch.empty(shape, device=a.device, dtype=torch.float32)
    n = len(shape)
    LL = ctypes.c_longlong * max(n, 1)
    _lib.check(_lib.cuda().fb_binary_fwd(ae.data_ptr(), be.data_ptr(), out.data_ptr(), BINARY[op], n,
                                         LL(*shape) if n else LL(1), LL(*ae.stride()) if n else LL(0),
                                         LL(*be.stride()) if n else LL(0), _stream()), "fb_binary_fwd")
    return out


_scratch_cache: dict = {}


def _scratch(device, nfloats: int) -> torch.Tensor:
    """A per-device fp32 workspace reused by reductions (grown on demand)."""
    key = (device.type, device.index)
    buf = _scratch_cache.get(key)
    if buf is None or buf.numel() < nfloats:
        buf = torch.empty(max(nfloats, 1 << 16), device=device, dtype=torch.float32)
        _scratch_cache[key] = buf
    return buf


def raw_reduce(x: torch.Tensor, op: str, dim: int | None, keepdim: bool = False) -> torch.Tensor:
    x = x.contiguous()
    if dim is None:
        outer, R, inner = 1, x.numel(), 1
        oshape = [1] * x.dim() if keepdim else []
    else:
        shp = list(x.shape)
        outer = math.prod(shp[:dim])
        R = shp[dim]
        inner = math.prod(shp[dim + 1:])
        oshape = shp[:dim] + ([1] if keepdim else []) + shp[dim + 1:]
    out = torch.empty(oshape, device=x.device, dtype=torch.float32)
    if out.numel() == 0:
        return out
    lib = _lib.cuda()
    want = lib.fb_reduce_scratch_elems(outer, R, inner)
    scr = _scratch(x.device, want) if want > 0 else None
    _lib.check(lib.fb_reduce(x.data_ptr(), out.data_ptr(), outer, R, inner, REDUCE[op], _ptr(scr),
                             scr.numel() if scr is not None else 0, _stream()), "fb_reduce")
    return out


def raw_colsum(x2d: torch.Tensor, out: torch.Tensor | None = None, accumulate: bool = False) -> torch.Tensor:
    x2d = x2d.contiguous()
    rows, cols = x2d.shape
    if out is None:
        out = torch.empty(cols, device=x2d.device, dtype=torch.float32)
        accumulate = False
    _lib.check(_lib.cuda().fb_colsum(x2d.data_ptr(), out.data_ptr(), rows, cols, _dt(x2d), 1 if accumulate else 0,
                                     _stream()), "fb_colsum")
    return out


def _f32(x: torch.Tensor) -> torch.Tensor:
    return raw_cast(x, torch.float32) if x.is_cuda else x.float()


def reduce_to_shape(g: torch.Tensor, shape) -> torch.Tensor:
    """Sum a broadcast gradient back to the operand's shape (autograd_ops.rs:589-640)."""
    shape = tuple(shape)
    if tuple(g.shape) == shape:
        return g
    if not g.is_cuda:
        return g.sum_to_size(shape) if shape else g.sum()
    out = _f32(g)
    while out.dim() > len(shape):
        out = raw_reduce(out, "sum", 0)
    for i, s in enumerate(shape):
        if s == 1 and out.shape[i] != 1:
            out = raw_reduce(out, "sum", i, keepdim=True)
    return out


# =============================================================================== elementwise
def _unary_cpu(x, op, a, b):
    if op == "relu":
        return torch.relu(x)
    if op == "gelu":
        return 0.5 * x * (1.0 + torch.tanh(GELU_C * (x + GELU_A * x * x * x)))
    if op == "silu":
        return x * torch.sigmoid(x)
    if op == "tanh":
        return torch.tanh(x)
    if op == "sigmoid":
        return torch.sigmoid(x)
    if op == "leaky_relu":
        return torch.where(x > 0, x, x * a)
    if op == "elu":
        return torch.where(x > 0, x, a * (torch.exp(x) - 1.0))
    if op == "neg":
        return -x
    if op == "exp":
        return torch.exp(x)
    if op == "log":
        return torch.log(x)
    if op == "sqrt":
        return torch.sqrt(x)
    if op == "abs":
        return torch.abs(x)
    if op == "sin":
        return torch.sin(x)
    if op == "cos":
        return torch.cos(x)
    if op == "pow":
        return torch.pow(x, a)
    if op == "add_scalar":
        return x + a
    if op == "mul_scalar":
        return x * a
    if op == "rsub_scalar":
        return a - x
    if op == "rdiv_scalar":
        return a / x
    if op == "affine":
        return x * a + b
    if op == "clamp":
        return torch.clamp(x, a, b)
    if op == "none":
        return x
    raise ValueError(op)


def unary(x: torch.Tensor, op: str, alpha: float = 0.0, beta: float = 0.0) -> torch.Tensor:
    if _native(x):
        return _lib.native().unary(x, UNARY[op], alpha, beta)
    return _unary_cpu(x, op, alpha, beta)


_SCALAR_TO_UNARY = {"add": "add_scalar", "mul": "mul_scalar", "rsub": "rsub_scalar", "rdiv": "rdiv_scalar"}


def scalar_op(x: torch.Tensor, op: str, s: float) -> torch.Tensor:
    """x (op) s for op in add / sub / mul / div / pow / rsub / rdiv — differentiable (unlike tensor.rs:1551-1591)."""
    if op == "sub":
        op, s = "add", -s
    elif op == "div":
        op, s = "mul", 1.0 / s
    if op == "pow":
        return unary(x, "pow", s)
    if op in ("max", "min"):
        return unary(x, "clamp", s if op == "max" else -3.0e38, 3.0e38 if op == "max" else s)
    return unary(x, _SCALAR_TO_UNARY[op], s)


class _BinaryFn(Function):
    @staticmethod
    def forward(ctx, a, b, op):
        af, bf = _f32(a), _f32(b)
        out = raw_binary(af, bf, op)
        ctx.op = op
        ctx.dtypes = (a.dtype, b.dtype)
        ctx.shapes = (a.shape, b.shape)
        if op in ("add", "sub"):
            ctx.save_for_backward()
        elif op in ("pow",):
            ctx.save_for_backward(af, bf, out)
        else:
            ctx.save_for_backward(af, bf)
        rd = torch.promote_types(a.dtype, b.dtype)
        return raw_cast(out, rd)

    @staticmethod
    def backward(ctx, g):
        op = ctx.op
        g = _f32(g.contiguous())
        need_a, need_b = ctx.needs_input_grad[0], ctx.needs_input_grad[1]
        ga = gb = None
        if op in ("add", "sub"):
            if need_a:
                ga = g
            if need_b:
                gb = g if op == "add" else raw_unary(g, "neg")
        else:
            a, b = ctx.saved_tensors[0], ctx.saved_tensors[1]
            if op == "mul":
                ga = raw_binary(g, b, "mul") if need_a else None
                gb = raw_binary(g, a, "mul") if need_b else None
            elif op == "div":
                ga = raw_binary(g, b, "div") if need_a else None
                if need_b:
                    q = raw_binary(raw_binary(g, a, "mul"), raw_binary(b, b, "mul"), "div")
                    gb = raw_unary(q, "neg")
            elif op == "pow":
                out = ctx.saved_tensors[2]
                if need_a:  # b * a^(b-1) = b * out / a
                    ga = raw_binary(g, raw_binary(raw_binary(b, out, "mul"), a, "div"), "mul")
                if need_b:
                    gb = raw_binary(g, raw_binary(out, raw_unary(a, "log"), "mul"), "mul")
            else:  # max / min: gradient goes to the selected operand (ties -> a)
                sel = (a >= b) if op == "max" else (a <= b)
                self_mask = sel.to(torch.float32)
                if need_a:
                    ga = raw_binary(g, self_mask, "mul")
                if need_b:
                    gb = raw_binary(g, raw_unary(self_mask, "rsub_scalar", 1.0), "mul")
        if ga is not None:
            ga = raw_cast(reduce_to_shape(ga, ctx.shapes[0]), ctx.dtypes[0])
        if gb is not None:
            gb = raw_cast(reduce_to_shape(gb, ctx.shapes[1]), ctx.dtypes[1])
        return ga, gb, None


def _binary_cpu(a, b, op):
    if op == "add":
        return a + b
    if op == "sub":
        return a - b
    if op == "mul":
        return a * b
    if op == "div":
        return a / b
    if op == "pow":
        return torch.pow(a, b)
    if op == "max":
        return torch.maximum(a, b)
    if op == "min":
        return torch.minimum(a, b)
    raise ValueError(op)


def binary(a: torch.Tensor, b: torch.Tensor, op: str) -> torch.Tensor:
    if _native(a) and _native(b):
        if op == "add" and a.shape == b.shape:
            return _lib.native().add(a, b)
        return _BinaryFn.apply(a, b, op)
    return _binary_cpu(a, b, op)


class _CastFn(Function):
    @staticmethod
    def forward(ctx, x, dtype):
        ctx.src = x.dtype
        return raw_cast(x, dtype)

    @staticmethod
    def backward(ctx, g):
        return raw_cast(g, ctx.src), None


def cast(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    if x.dtype == dtype:
        return x
    if x.is_cuda and {x.dtype, dtype} == {torch.float32, torch.bfloat16}:
        return _CastFn.apply(x, dtype)
    return x.to(dtype)


def cat(tensors, dim: int = 0) -> torch.Tensor:
    """Concatenation is pure data movement (async device copies); torch provides the CatBackward split."""
    return torch.cat(list(tensors), dim)


# =============================================================================== reductions
class _ReduceFn(Function):
    @staticmethod
    def forward(ctx, x, op, dim, keepdim):
        xf = _f32(x)
        y = raw_reduce(xf, op, dim, True)
        ctx.op, ctx.dim, ctx.keepdim, ctx.src_dtype = op, dim, keepdim, x.dtype
        ctx.xshape = x.shape
        if op in ("max", "min", "prod"):
            ctx.save_for_backward(xf, y)
        else:
            ctx.save_for_backward()
        out = y if keepdim else (y.reshape(()) if dim is None else y.squeeze(dim))
        return raw_cast(out, x.dtype)

    @staticmethod
    def backward(ctx, g):
        op, dim = ctx.op, ctx.dim
        g = _f32(g)
        kshape = [1] * len(ctx.xshape) if dim is None else [
            1 if i == dim else s for i, s in enumerate(ctx.xshape)]
        gk = g.reshape(kshape)
        if op == "sum":
            gx = gk.expand(ctx.xshape)
        elif op == "mean":
            R = math.prod(ctx.xshape) if dim is None else ctx.xshape[dim]
            gx = raw_unary(gk, "mul_scalar", 1.0 / max(R, 1)).expand(ctx.xshape)
        elif op in ("max", "min"):
            x, y = ctx.saved_tensors
            mask = (x == y).to(torch.float32)
            gx = raw_binary(gk, mask, "mul")
        else:  # prod: d/dx_i = prod / x_i
            x, y = ctx.saved_tensors
            gx = raw_binary(raw_binary(gk, y, "mul"), x, "div")
        if gx.dtype != ctx.src_dtype:
            gx = raw_cast(gx.contiguous(), ctx.src_dtype)
        return gx, None, None, None


def reduce(x: torch.Tensor, op: str, dim: int | None = None, keepdim: bool = False) -> torch.Tensor:
    if _native(x) and x.numel() > 0:
        return _ReduceFn.apply(x, op, dim, keepdim)
    if dim is None:
        fn = {"sum": torch.sum, "mean": torch.mean, "max": torch.max, "min": torch.min, "prod": torch.prod}[op]
        out = fn(x)
        return out.reshape([1] * x.dim()) if keepdim else out
    if op in ("max", "min"):
        return getattr(torch, op)(x, dim=dim, keepdim=keepdim).values
    return getattr(torch, op)(x, dim=dim, keepdim=keepdim)


def arg_reduce(x: torch.Tensor, is_max: bool, dim: int | None = None, keepdim: bool = False) -> torch.Tensor:
    """Index of the first maximum / minimum (tensor.rs:1838-2036)."""
    if _native(x) and x.numel() > 0:
        xf = _f32(x).contiguous()
        if dim is None:
            outer, R, inner, oshape = 1, xf.numel(), 1, []
        else:
            shp = list(xf.shape)
            outer, R, inner = math.prod(shp[:dim]), shp[dim], math.prod(shp[dim + 1:])
            oshape = shp[:dim] + ([1] if keepdim else []) + shp[dim + 1:]
        idx = torch.empty(oshape, device=x.device, dtype=torch.int64)
        _lib.check(_lib.cuda().fb_arg_reduce(xf.data_ptr(), idx.data_ptr(), None, outer, R, inner,
                                             1 if is_max else 0, _stream()), "fb_arg_reduce")
        return idx
    fn = torch.argmax if is_max else torch.argmin
    return fn(x) if dim is None else fn(x, dim=dim, keepdim=keepdim)


# =============================================================================== GEMM-shaped ops
def _gemm_nt(a: torch.Tensor, b_nt: torch.Tensor, bias=None, act=None, low: bool = False, out=None,
             out_dtype=None, accumulate=False) -> torch.Tensor:
    """out = act(a @ b_nt^T + bias) with a [M,K], b_nt [N,K] (any strides)."""
    dt = torch.bfloat16 if low else torch.float32
    ab = a if a.dtype == dt else raw_cast(a.contiguous(), dt)
    bb = b_nt if b_nt.dtype == dt else raw_cast(b_nt.contiguous(), dt)
    if out is None:
        out = torch.empty((a.shape[0], b_nt.shape[0]), device=a.device, dtype=out_dtype or dt)
        accumulate = False
    _lib.native().gemm_nt(ab, bb, bias, _gemm.ACT[act], out, accumulate, not low and config.tf32_active())
    return out


class _MatmulFn(Function):
    @staticmethod
    def forward(ctx, a, b, low):
        ctx.low = low
        ctx.dtypes = (a.dtype, b.dtype)
        if low:
            a = raw_cast(a.contiguous(), torch.bfloat16)
            b = raw_cast(b.contiguous(), torch.bfloat16)
        ctx.save_for_backward(a, b)
        out = _gemm_nt(a, b.t(), low=low)
        return out if low else raw_cast(out, torch.promote_types(*ctx.dtypes))

    @staticmethod
    def backward(ctx, g):
        a, b = ctx.saved_tensors
        low = ctx.low
        g = g.contiguous()
        if low and g.dtype != torch.bfloat16:
            g = raw_cast(g, torch.bfloat16)
        ga = gb = None
        if ctx.needs_input_grad[0]:
            ga = raw_cast(_gemm_nt(g, b, low=low), ctx.dtypes[0])
        if ctx.needs_input_grad[1]:
            gb = raw_cast(_gemm_nt(a.t(), g.t(), low=low, out_dtype=torch.float32), ctx.dtypes[1])
        return ga, gb, None


def bmm_scaled(a: torch.Tensor, b: torch.Tensor, alpha: float = 1.0, heads_inner: bool = False) -> torch.Tensor:
    """``alpha * a @ b`` for 4-D ``[Bo, Bi, M, K] @ [Bo, Bi, K, N]``: tensor cores under autocast for TMA-describable
    operands (feature extents multiples of 8), the fp32 batched kernel otherwise.  ``heads_inner`` stores the
    result as ``[Bo, M, Bi, N]`` (returned as the permuted view)."""
    if _native(a) and _native(b):
        low = config.low_precision_active()
        if (a.shape[-1] % 8 == 0 and b.shape[-1] % 8 == 0) if low else (
                a.dim() == b.dim() == 4 and a.dtype == b.dtype == torch.float32 and a.shape[:2] == b.shape[:2]):
            return _lib.native().bmm(a, b, alpha, heads_inner, low)
    out = matmul(a, b)
    return scalar_op(out, "mul", float(alpha)) if alpha != 1.0 else out


def flash_attention_ok(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, need_no_grad: bool = True,
                       head_dims=(64, 128)) -> bool:
    """True when ``flash_attention`` can take these ``[B, H, S, D]`` operands: CUDA, head dimension 64 or 128
    (``head_dims``) contiguous, other strides multiples of 8 elements and (``need_no_grad``) no gradient needed —
    the kernel records no autograd node."""
    if not (q.is_cuda and q.dim() == 4 and k.dim() == 4 and v.dim() == 4 and q.shape[-1] in head_dims):
        return False
    D = q.shape[-1]
    if need_no_grad and torch.is_grad_enabled() and (q.requires_grad or k.requires_grad or v.requires_grad):
        return False
    if k.shape != v.shape or q.shape[:2] != k.shape[:2] or k.shape[-1] != D:
        return False
    for t in (q, k, v):
        if t.stride(-1) != 1 or any(s % 8 for s in t.stride()[:-1]) or t.stride(2) < D:
            return False
    return True


def flash_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float,
                    return_lse: bool = False, causal: bool = False):
    """``softmax(scale * q @ k^T) @ v`` for ``[B, H, S, D]`` operands (D = 64 or 128) without materialising the
    score matrix: one tcgen05 kernel with online softmax (csrc/kernels/attention.cu).  No autograd node is recorded
    here (:func:`attention_blockwise` is the differentiable form).  ``causal``: query ``i`` sees
    keys ``j <= i + (Skv - Sq)`` and key tiles past the diagonal are skipped.  The result is stored as
    ``[B, Sq, H, D]`` and returned as the ``[B, H, Sq, D]`` view (like ``bmm_scaled(..., heads_inner=True)``)."""
    B, H, Sq, D = q.shape
    Skv = k.shape[2]
    qb, kb, vb = (t if t.dtype == torch.bfloat16 else t.to(torch.bfloat16) for t in (q.detach(), k.detach(), v.detach()))
    out = torch.empty((B, Sq, H, D), device=q.device, dtype=torch.bfloat16)
    lse = torch.empty((B, H, Sq), device=q.device, dtype=torch.float32) if return_lse else None
    rc = _lib.cuda().fb_attention_fwd(qb.data_ptr(), kb.data_ptr(), vb.data_ptr(), out.data_ptr(),
                                      lse.data_ptr() if lse is not None else None, B, H, Sq, Skv, D,
                                      qb.stride(0), qb.stride(1), qb.stride(2), kb.stride(0), kb.stride(1),
                                      kb.stride(2), vb.stride(0), vb.stride(1), vb.stride(2), float(scale),
                                      1 if causal else 0, _rt.status_ptr(), _stream())
    _lib.check(rc, "fb_attention_fwd")
    res = out.permute(0, 2, 1, 3)
    return (res, lse) if return_lse else res


class _BlockwiseAttentionFn(Function):
    """``softmax(scale q k^T) v`` with the blockwise tcgen05 kernels in BOTH directions: the forward saves q, k, v,
    the output and one log-sum-exp per row; the backward recomputes the probabilities tile by tile
    (csrc/kernels/attention_bwd.cu).  Nothing of size S x S is ever stored."""

    @staticmethod
    def forward(ctx, q, k, v, scale, causal):
        out, lse = flash_attention(q, k, v, scale, return_lse=True, causal=causal)
        qb, kb, vb = (t if t.dtype == torch.bfloat16 else t.to(torch.bfloat16) for t in (q, k, v))
        ctx.save_for_backward(qb, kb, vb, out, lse)
        ctx.scale, ctx.causal = scale, causal
        ctx.in_dtypes = (q.dtype, k.dtype, v.dtype)
        return out

    @staticmethod
    def backward(ctx, g):
        q, k, v, out, lse = ctx.saved_tensors
        B, H, Sq, D = q.shape
        Skv = k.shape[2]
        o = out.permute(0, 2, 1, 3)                      # the kernel's own [B, Sq, H, D] storage
        if not o.is_contiguous():
            o = o.contiguous()
        go = g.permute(0, 2, 1, 3)
        if go.dtype != torch.bfloat16 or not go.is_contiguous():
            go = go.to(torch.bfloat16).contiguous()
        dq = torch.empty((B, Sq, H, D), device=q.device, dtype=torch.bfloat16)
        dk = torch.empty((B, Skv, H, D), device=q.device, dtype=torch.bfloat16)
        dv = torch.empty((B, Skv, H, D), device=q.device, dtype=torch.bfloat16)
        delta = torch.empty((B, H, Sq), device=q.device, dtype=torch.float32)
        rc = _lib.cuda().fb_attention_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), go.data_ptr(),
                                          lse.data_ptr(), delta.data_ptr(), dq.data_ptr(), dk.data_ptr(),
                                          dv.data_ptr(), B, H, Sq, Skv, D, q.stride(0), q.stride(1), q.stride(2),
                                          k.stride(0), k.stride(1), k.stride(2), v.stride(0), v.stride(1),
                                          v.stride(2), float(ctx.scale), 1 if ctx.causal else 0, _rt.status_ptr(),
                                          _stream())
        if -5 <= rc <= -2:  # an operand that no TMA map describes: name it
            name, t = {-2: ("q", q), -3: ("k", k), -4: ("v", v), -5: ("grad_output", go)}[rc]
            raise ValueError(f"fb_attention_bwd: {name} of shape {tuple(t.shape)}, strides {t.stride()}, address "
                             f"{t.data_ptr():#x} cannot be a TMA operand (16-byte aligned pointer, strides multiples of 8; "
                             f"reason {_lib.cuda().fb_attention_bwd_map_error()})")
        _lib.check(rc, "fb_attention_bwd")
        grads = [t.permute(0, 2, 1, 3) for t in (dq, dk, dv)]
        grads = [gr if gr.dtype == dt else gr.to(dt) for gr, dt in zip(grads, ctx.in_dtypes)]
        return grads[0], grads[1], grads[2], None, None


def attention_blockwise(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float,
                        causal: bool = False) -> torch.Tensor:
    """Differentiable blockwise attention for ``[B, H, S, D]`` operands, D = 64 or 128 (see ``flash_attention_ok``):
    forward and backward on the tcgen05 kernels, no S x S matrix in memory in either direction."""
    return _BlockwiseAttentionFn.apply(q, k, v, float(scale), bool(causal))


class _CheckpointedAttentionFn(Function):
    """Attention core with the blockwise kernel in the forward pass and NOTHING of size S x S kept for the backward
    pass: the backward recomputes the scores with the differentiable batched-GEMM path (activation checkpointing
    of the attention core).  Trades one extra score computation for S x S x heads of saved activations."""

    @staticmethod
    def forward(ctx, q, k, v, scale):
        ctx.scale = scale
        ctx.save_for_backward(q, k, v)
        return flash_attention(q, k, v, scale)

    @staticmethod
    def backward(ctx, g):
        q, k, v = ctx.saved_tensors
        # the backward pass runs outside the caller's autocast block: re-enter it for the recomputation
        with torch.enable_grad(), config.autocast():
            qd, kd, vd = (t.detach().requires_grad_(True) for t in (q, k, v))
            attn = softmax(bmm_scaled(qd, kd.transpose(-1, -2), ctx.scale), -1)
            out = bmm_scaled(attn, vd, 1.0, heads_inner=True)
            gq, gk, gv = torch.autograd.grad(out, (qd, kd, vd), g.to(out.dtype))
        return gq, gk, gv, None


def attention_checkpointed(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float) -> torch.Tensor:
    """Differentiable ``softmax(scale q k^T) v`` that saves only q, k, v (see ``_CheckpointedAttentionFn``);
    operands as for :func:`flash_attention`."""
    return _CheckpointedAttentionFn.apply(q, k, v, float(scale))


def matmul(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """2D@2D, 2D@1D, 1D@2D (tensor.rs:2433-2485) and batched ND@ND / ND@2D."""
    if not (_native(a) and _native(b)):
        return torch.matmul(a, b)
    low = config.low_precision_active()
    if a.dim() == 1 and b.dim() == 1:
        return reduce(binary(a, b, "mul"), "sum")
    if a.dim() == 1:
        return matmul(a.unsqueeze(0), b).squeeze(-2)
    if b.dim() == 1:
        return matmul(a, b.unsqueeze(1)).squeeze(-1)
    if a.dim() == 2 and b.dim() == 2:
        return _MatmulFn.apply(a, b, low)
    if b.dim() == 2:  # [..., M, K] @ [K, N]
        lead = a.shape[:-1]
        return _MatmulFn.apply(a.reshape(-1, a.shape[-1]), b, low).reshape(*lead, b.shape[1])
    # batched: broadcast batch dims; tensor cores under autocast, else the fp32 batched kernel
    bs = torch.broadcast_shapes(a.shape[:-2], b.shape[:-2])
    if low and a.shape[-1] % 8 == 0 and b.shape[-1] % 8 == 0:
        a4 = a.expand(*bs, *a.shape[-2:]).reshape(1, -1, *a.shape[-2:])
        b4 = b.expand(*bs, *b.shape[-2:]).reshape(1, -1, *b.shape[-2:])
        return _lib.native().bmm(a4, b4, 1.0, False, True).reshape(*bs, a.shape[-2], b.shape[-1])
    a4 = _f32(a.expand(*bs, *a.shape[-2:])).reshape(1, -1, *a.shape[-2:])
    b4 = _f32(b.expand(*bs, *b.shape[-2:])).reshape(1, -1, *b.shape[-2:])
    out = _lib.native().bmm(a4, b4, 1.0, False, False)
    return raw_cast(out.reshape(*bs, a.shape[-2], b.shape[-1]), torch.promote_types(a.dtype, b.dtype))


class GradSink:
    """Where a Linear's weight gradient is written.

    ``acquire(param)`` returns ``(buffer, accumulate)``: an fp32 tensor shaped like
    the parameter and whether the wgrad GEMM must add to its contents; ``ready(param)``
    is called once the gradient is enqueued on the current stream.  The DDP engine
    implements this to have wgrad written straight into its flat gradient arena.
    """

    def acquire(self, param):  # pragma: no cover - interface
        raise NotImplementedError

    def ready(self, param):  # pragma: no cover - interface
        raise NotImplementedError


_FUSABLE_ACT = {"relu", "tanh", "sigmoid"}  # derivative expressible from the output


def linear(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor | None = None, act: str | None = None,
           w_low: torch.Tensor | None = None, sink: GradSink | None = None) -> torch.Tensor:
    """``act(x @ weight^T + bias)`` with weight ``[out, in]`` (ferrum-nn/src/linear.rs:78-89).

    On CUDA the bias (and relu/tanh/sigmoid) run in the GEMM epilogue.  ``w_low`` is an
    up-to-date bf16 copy of ``weight`` (kept by the optimizer) used under bf16 precision.
    """
    if not _native(x):
        y = torch.nn.functional.linear(x, weight, bias)
        return _unary_cpu(y, act, 0.0, 0.0) if act else y
    low = config.low_precision_active()
    tf32 = not low and config.tf32_active()
    if act is not None and act not in _FUSABLE_ACT and torch.is_grad_enabled() and (
            x.requires_grad or weight.requires_grad or (bias is not None and bias.requires_grad)):
        return unary(_lib.native().linear(x, weight, bias, 0, low, tf32, w_low, sink), act)
    # the activations a GEMM epilogue evaluates; another name is a KeyError
    return _lib.native().linear(x, weight, bias, _gemm.ACT[act], low, tf32, w_low, sink)


# =============================================================================== normalisation
def layer_norm(x: torch.Tensor, gamma=None, beta=None, eps: float = 1e-5, pre_act: str | None = None,
               n_norm_dims: int = 1) -> torch.Tensor:
    """Normalise over the last ``n_norm_dims`` dimensions; optional fused GELU before the statistics."""
    if n_norm_dims != 1:
        lead = x.shape[:-n_norm_dims]
        flat = x.reshape(*lead, -1)
        g = gamma.reshape(-1) if gamma is not None else None
        b = beta.reshape(-1) if beta is not None else None
        return layer_norm(flat, g, b, eps, pre_act, 1).reshape(x.shape)
    if _native(x):
        return _lib.native().layer_norm(x, gamma, beta, eps, UNARY[pre_act or "none"])
    a = _unary_cpu(x, pre_act, 0.0, 0.0) if pre_act else x
    mu = a.mean(-1, keepdim=True)
    var = ((a - mu) ** 2).mean(-1, keepdim=True)
    y = (a - mu) / torch.sqrt(var + eps)
    if gamma is not None:
        y = y * gamma
    if beta is not None:
        y = y + beta
    return y


def add_layer_norm(x, r, gamma=None, beta=None, eps: float = 1e-5):
    """``layer_norm(x + r)`` over the last dimension as one node (tensors of one size)."""
    if _native(x) and _native(r) and x.shape == r.shape:
        return _lib.native().add_layer_norm(x, r, gamma, beta, eps)
    return layer_norm(binary(x, r, "add"), gamma, beta, eps)


def linear_act_layernorm(x, weight, bias, gamma, beta, eps: float = 1e-5, act: str = "gelu", w_low=None,
                         sink: GradSink | None = None):
    """``LayerNorm(act(x @ weight^T + bias)) * gamma + beta`` as one fused block (CUDA); composed ops on CPU."""
    if _native(x) and gamma is not None and beta is not None:
        low = config.low_precision_active()
        return _lib.native().linear_act_norm(x, weight, bias, gamma, beta, eps, UNARY[act or "none"], low,
                                             not low and config.tf32_active(), w_low, sink)
    return layer_norm(linear(x, weight, bias, None, w_low, sink), gamma, beta, eps, act)


class _BatchNormFn(Function):
    @staticmethod
    def forward(ctx, x, gamma, beta, running_mean, running_var, eps, momentum, training):
        x2 = _f32(x).contiguous()
        rows, cols = x2.shape
        y = torch.empty_like(x2)
        sm = torch.empty(cols, device=x.device, dtype=torch.float32)
        sr = torch.empty(cols, device=x.device, dtype=torch.float32)
        g = gamma.detach().contiguous() if gamma is not None else None
        b = beta.detach().contiguous() if beta is not None else None
        _lib.check(_lib.cuda().fb_batchnorm_fwd(x2.data_ptr(), _ptr(g), _ptr(b), y.data_ptr(), sm.data_ptr(),
                                                sr.data_ptr(), _ptr(running_mean), _ptr(running_var), rows, cols,
                                                eps, momentum, 1 if training else 0, _stream()),
                   "fb_batchnorm_fwd")
        if not training:
            sm = running_mean.detach().clone()
            sr = torch.rsqrt(running_var.detach() + eps)
        ctx.save_for_backward(x2, g, sm, sr)
        ctx.training = training
        ctx.flags = (gamma is not None, beta is not None)
        ctx.src_dtype = x.dtype
        return raw_cast(y, x.dtype)

    @staticmethod
    def backward(ctx, gy):
        x2, g, sm, sr = ctx.saved_tensors
        rows, cols = x2.shape
        gy2 = _f32(gy).contiguous()
        if ctx.training:
            dx = torch.empty_like(x2)
            dgamma = torch.empty(cols, device=x2.device, dtype=torch.float32)
            dbeta = torch.empty(cols, device=x2.device, dtype=torch.float32)
            _lib.check(_lib.cuda().fb_batchnorm_bwd(gy2.data_ptr(), x2.data_ptr(), _ptr(g), sm.data_ptr(),
                                                    sr.data_ptr(), dx.data_ptr(), dgamma.data_ptr(),
                                                    dbeta.data_ptr(), rows, cols, _stream()), "fb_batchnorm_bwd")
        else:  # statistics are constants in eval mode
            scale = sr if g is None else raw_binary(sr, g, "mul")
            dx = raw_binary(gy2, scale, "mul")
            xhat = raw_binary(raw_binary(x2, sm, "sub"), sr, "mul")
            dgamma = raw_reduce(raw_binary(gy2, xhat, "mul"), "sum", 0)
            dbeta = raw_reduce(gy2, "sum", 0)
        return (raw_cast(dx, ctx.src_dtype), dgamma if ctx.flags[0] else None, dbeta if ctx.flags[1] else None,
                None, None, None, None, None)


def batch_norm(x: torch.Tensor, gamma, beta, running_mean, running_var, training: bool, momentum: float = 0.1,
               eps: float = 1e-5) -> torch.Tensor:
    """Per-feature batch normalisation of ``[B, F]`` input with running-stat update."""
    if x.dim() != 2:
        raise ValueError("batch_norm expects [batch, features]")
    if _native(x):
        return _BatchNormFn.apply(x, gamma, beta, running_mean, running_var, float(eps), float(momentum),
                                  bool(training))
    if training:
        mu = x.mean(0)
        var = ((x - mu) ** 2).mean(0)
        if running_mean is not None:
            with torch.no_grad():
                n = x.shape[0]
                running_mean.mul_(1 - momentum).add_(momentum * mu.detach())
                running_var.mul_(1 - momentum).add_(momentum * var.detach() * (n / (n - 1) if n > 1 else 1.0))
    else:
        mu, var = running_mean, running_var
    y = (x - mu) / torch.sqrt(var + eps)
    if gamma is not None:
        y = y * gamma
    if beta is not None:
        y = y + beta
    return y


# =============================================================================== softmax / losses
def _softmax_any_dim(x, dim, log_mode):
    nd = x.dim()
    if nd == 0:
        x = x.reshape(1)
        nd, dim = 1, 0
    d = dim + nd if dim < 0 else dim
    if _native(x):
        if d != nd - 1:
            return _lib.native().softmax(x.transpose(d, -1), log_mode).transpose(d, -1)
        return _lib.native().softmax(x, log_mode)
    return torch.log_softmax(x, d) if log_mode else torch.softmax(x, d)


def softmax(x: torch.Tensor, dim: int = -1) -> torch.Tensor:
    """Numerically stable softmax along ``dim`` (per-row spec of ferrum-cuda/src/kernels.rs:501-560)."""
    return _softmax_any_dim(x, dim, False)


def log_softmax(x: torch.Tensor, dim: int = -1) -> torch.Tensor:
    return _softmax_any_dim(x, dim, True)


def cross_entropy_logits(logits: torch.Tensor, labels: torch.Tensor) -> torch.Tensor:
    """Mean over the batch of ``-log softmax(logits)[label]`` for integer ``labels`` (fused kernel on CUDA)."""
    if logits.dim() != 2:
        logits = logits.reshape(-1, logits.shape[-1])
        labels = labels.reshape(-1)
    labels = labels.to(torch.int64)
    if _native(logits):
        return _lib.native().cross_entropy(logits, labels)
    lp = torch.log_softmax(logits.float(), -1)
    return -lp.gather(1, labels.unsqueeze(1)).mean()


def nll_index(log_probs: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
    """Mean over the rows of ``-log_probs[i, targets[i]]`` for integer ``targets`` on the GPU."""
    return _lib.native().nll(log_probs, targets)


def elementwise_loss(pred: torch.Tensor, target: torch.Tensor, kind: str) -> torch.Tensor:
    """mse / bce / l1 / smooth_l1, mean over all elements (ferrum-nn/src/loss.rs:24-105)."""
    if tuple(pred.shape) != tuple(target.shape):
        target = target.expand_as(pred)
    if _native(pred) and pred.numel() > 0:
        return _lib.native().elementwise_loss(pred, target, LOSS[kind])
    d = pred - target
    if kind == "mse":
        return (d * d).mean()
    if kind == "bce":
        eps = 1e-7
        pc = pred + eps
        q = (1.0 + eps) - pc
        return -(target * torch.log(pc) + (1.0 - target) * torch.log(q)).mean()
    if kind == "l1":
        return d.abs().mean()
    a = d.abs()
    return torch.where(a < 1.0, 0.5 * d * d, a - 0.5).mean()


# =============================================================================== dropout / embedding / gather
_dropout_offset = 0


_capturable_rng = {}  # device index -> uint64 counter tensor; non-empty while steps are recorded in CUDA graphs


def set_capturable_rng(flag: bool) -> None:
    """Draw dropout offsets from a device-side counter that advances on the stream, so a step recorded in a CUDA
    graph draws a new mask at every replay (a host-side counter would be frozen into the graph)."""
    if not flag:
        _capturable_rng.clear()
    elif torch.cuda.is_available() and torch.cuda.current_device() not in _capturable_rng:
        _capturable_rng[torch.cuda.current_device()] = torch.zeros(1, dtype=torch.int64, device="cuda")


class _DropoutFn(Function):
    @staticmethod
    def forward(ctx, x, p, seed, offset):
        x2 = x.contiguous()
        y = torch.empty_like(x2)
        mask = torch.empty(x2.shape, device=x.device, dtype=torch.uint8)
        ctr = _capturable_rng.get(x.device.index)
        if ctr is not None:
            _lib.check(_lib.cuda().fb_dropout_fwd_dyn(x2.data_ptr(), y.data_ptr(), mask.data_ptr(), x2.numel(), p,
                                                      seed, offset << 20, ctr.data_ptr(), _dt(x2), _stream()),
                       "fb_dropout_fwd_dyn")
        else:
            _lib.check(_lib.cuda().fb_dropout_fwd(x2.data_ptr(), y.data_ptr(), mask.data_ptr(), x2.numel(), p, seed,
                                                  offset, _dt(x2), _stream()), "fb_dropout_fwd")
        ctx.save_for_backward(mask)
        ctx.p = p
        return y

    @staticmethod
    def backward(ctx, g):
        (mask,) = ctx.saved_tensors
        g2 = g.contiguous()
        dx = torch.empty_like(g2)
        _lib.check(_lib.cuda().fb_dropout_bwd(g2.data_ptr(), mask.data_ptr(), dx.data_ptr(), g2.numel(), ctx.p,
                                              _dt(g2), _stream()), "fb_dropout_bwd")
        return dx, None, None, None


def dropout(x: torch.Tensor, p: float, training: bool, seed: int | None = None) -> torch.Tensor:
    """Inverted dropout: keep with probability 1-p and scale by 1/(1-p) while training; identity otherwise."""
    global _dropout_offset
    if not training or p <= 0.0:
        return x
    if p >= 1.0:
        return x * 0.0
    if _native(x):
        if seed is None:
            seed = torch.initial_seed()
        _dropout_offset += 1
        return _DropoutFn.apply(x, float(p), int(seed) & 0xFFFFFFFFFFFFFFFF, _dropout_offset)
    return torch.nn.functional.dropout(x, p, True)


def embedding(weight: torch.Tensor, idx: torch.Tensor, padding_idx: int | None = None,
              out_dtype: torch.dtype | None = None, sink: GradSink | None = None) -> torch.Tensor:
    """Row gather ``weight[idx]`` -> ``[*idx.shape, D]``; rows at ``padding_idx`` are zero (embedding.rs:122-208)."""
    idx = idx.to(torch.int64)
    if weight.is_cuda and weight.dtype == torch.float32:
        return _lib.native().embedding(weight, idx, -1 if padding_idx is None else padding_idx, False,
                                       out_dtype == torch.bfloat16, sink)
    out = torch.nn.functional.embedding(idx, weight)
    if padding_idx is not None:
        out = out * (idx != padding_idx).unsqueeze(-1).to(out.dtype)
    return out


def embedding_mean_pool(weight: torch.Tensor, idx: torch.Tensor, out_dtype: torch.dtype | None = None,
                        sink: GradSink | None = None):
    """``mean_s weight[idx[b, s]]`` for ``idx [B, S]`` without materialising ``[B, S, D]``."""
    idx = idx.to(torch.int64)
    if weight.is_cuda and weight.dtype == torch.float32 and idx.dim() == 2 and idx.shape[1] * 8 <= 48 * 1024:
        return _lib.native().embedding(weight, idx, -1, True, out_dtype == torch.bfloat16, sink)
    return torch.nn.functional.embedding(idx, weight).mean(1)


def gather_rows(src: torch.Tensor, idx: torch.Tensor) -> torch.Tensor:
    """``src[idx]`` along dim 0 for a contiguous device-resident tensor (DataLoader collate)."""
    if not src.is_cuda:
        return src.index_select(0, idx.to(torch.int64))
    src = src.contiguous()
    idx = idx.to(device=src.device, dtype=torch.int64).contiguous()
    out = torch.empty((idx.numel(), *src.shape[1:]), device=src.device, dtype=src.dtype)
    row_bytes = src[0].numel() * src.element_size() if src.shape[0] else 0
    if idx.numel() == 0 or row_bytes == 0:
        return out
    # an index outside the source is reported through the status block and its row comes back as zeros
    _lib.check(_lib.cuda().fb_gather_rows(src.data_ptr(), idx.data_ptr(), out.data_ptr(), idx.numel(), row_bytes,
                                          src.shape[0], _rt.status_ptr(), _stream()), "fb_gather_rows")
    return out


def transpose_2d(x: torch.Tensor) -> torch.Tensor:
    """Materialised transpose of a 2-D tensor (ferrum-cuda/src/kernels.rs:442-494)."""
    if not (x.is_cuda and x.element_size() in (2, 4)):
        return x.t().contiguous()
    x = x.contiguous()
    out = torch.empty((x.shape[1], x.shape[0]), device=x.device, dtype=x.dtype)
    _lib.check(_lib.cuda().fb_transpose_2d(x.data_ptr(), out.data_ptr(), x.shape[0], x.shape[1], x.element_size(),
                                           _stream()), "fb_transpose_2d")
    return out


# ============================================================ secondary layers: recurrent gates, conv lowering, pooling
class _LstmGatesFn(Function):
    """(h', c') from the gate pre-activations ``xi + hh`` ([B, 4H]: input, forget, cell, output) in one kernel."""

    @staticmethod
    def forward(ctx, xi, hh, c_prev):
        xi, hh, c_prev = _f32(xi).contiguous(), _f32(hh).contiguous(), _f32(c_prev).contiguous()
        B, H = c_prev.shape
        h, c = torch.empty_like(c_prev), torch.empty_like(c_prev)
        gates = torch.empty_like(xi)
        _lib.check(_lib.cuda().fb_lstm_gates_fwd(xi.data_ptr(), hh.data_ptr(), c_prev.data_ptr(), h.data_ptr(),
                                                 c.data_ptr(), gates.data_ptr(), B, H, _stream()), "fb_lstm_gates_fwd")
        ctx.save_for_backward(gates, c_prev, c)
        return h, c

    @staticmethod
    def backward(ctx, dh, dc):
        gates, c_prev, c = ctx.saved_tensors
        B, H = c_prev.shape
        dh = _f32(dh).contiguous() if dh is not None else None
        dc = _f32(dc).contiguous() if dc is not None else None
        dpre, dc_prev = torch.empty_like(gates), torch.empty_like(c_prev)
        _lib.check(_lib.cuda().fb_lstm_gates_bwd(dh.data_ptr() if dh is not None else None,
                                                 dc.data_ptr() if dc is not None else None, gates.data_ptr(),
                                                 c_prev.data_ptr(), c.data_ptr(), dpre.data_ptr(), dc_prev.data_ptr(),
                                                 B, H, _stream()), "fb_lstm_gates_bwd")
        return dpre, dpre, dc_prev


def lstm_gates(xi, hh, c_prev):
    """LSTM cell update from the two projections (ferrum-nn/src/rnn.rs:188-227)."""
    if _native(xi) and xi.dim() == 2:
        return _LstmGatesFn.apply(xi, hh, c_prev)
    i, f, g, o = (xi + hh).chunk(4, -1)
    c = torch.sigmoid(f) * c_prev + torch.sigmoid(i) * torch.tanh(g)
    return torch.sigmoid(o) * torch.tanh(c), c


class _GruGatesFn(Function):
    """h' = (1 - z) n + z h with r, z = sigmoid, n = tanh(xn + r * hn), from xi, hh [B, 3H] in one kernel."""

    @staticmethod
    def forward(ctx, xi, hh, h_prev):
        xi, hh, h_prev = _f32(xi).contiguous(), _f32(hh).contiguous(), _f32(h_prev).contiguous()
        B, H = h_prev.shape
        h = torch.empty_like(h_prev)
        saved = torch.empty((B, 4 * H), device=h.device, dtype=torch.float32)
        _lib.check(_lib.cuda().fb_gru_gates_fwd(xi.data_ptr(), hh.data_ptr(), h_prev.data_ptr(), h.data_ptr(),
                                                saved.data_ptr(), B, H, _stream()), "fb_gru_gates_fwd")
        ctx.save_for_backward(saved, h_prev)
        return h

    @staticmethod
    def backward(ctx, dh):
        saved, h_prev = ctx.saved_tensors
        B, H = h_prev.shape
        dh = _f32(dh).contiguous()
        dxi = torch.empty((B, 3 * H), device=dh.device, dtype=torch.float32)
        dhh, dhp = torch.empty_like(dxi), torch.empty_like(h_prev)
        _lib.check(_lib.cuda().fb_gru_gates_bwd(dh.data_ptr(), saved.data_ptr(), h_prev.data_ptr(), dxi.data_ptr(),
                                                dhh.data_ptr(), dhp.data_ptr(), B, H, _stream()), "fb_gru_gates_bwd")
        return dxi, dhh, dhp


def gru_gates(xi, hh, h_prev):
    """GRU cell update from the two projections (ferrum-nn/src/rnn.rs:318-372)."""
    if _native(xi) and xi.dim() == 2:
        return _GruGatesFn.apply(xi, hh, h_prev)
    xr, xz, xn = xi.chunk(3, -1)
    hr, hz, hn = hh.chunk(3, -1)
    r, z = torch.sigmoid(xr + hr), torch.sigmoid(xz + hz)
    n = torch.tanh(xn + r * hn)
    return (1 - z) * n + z * h_prev


def rnn_sequence_ok(gates: int, x: torch.Tensor, weight_hh: torch.Tensor) -> bool:
    """True when a whole layer's recurrence over ``x [T, B, F]`` can run in one launch per direction
    (csrc/kernels/rnn_seq.cu): fp32 on the GPU, the recurrent matrix within a cluster's shared memory."""
    return (x.is_cuda and x.dtype == weight_hh.dtype == torch.float32 and x.shape[0] > 0 and x.shape[1] > 0
            and not config.low_precision_active() and not config.tf32_active()
            and _lib.native().rnn_seq_supported(gates, x.shape[1], weight_hh.shape[1]))


def rnn_sequence(gates: int, proj, weight_hh, bias_hh, h0=None, c0=None):
    """``[hs]`` (GRU, gates = 3) or ``[hs, c_last]`` (LSTM, gates = 4) from the input projections ``[T, B, gates H]``;
    absent initial states are zero."""
    return _lib.native().rnn_seq(gates, proj, weight_hh, bias_hh, h0, c0)


def conv_out_size(size, k, stride, pad, dil):
    return (size + 2 * pad - dil * (k - 1) - 1) // stride + 1


class _Im2colFn(Function):
    """[B, C, H, W] -> window matrix [B*Ho*Wo, C*kh*kw], K contiguous: the A operand of the convolution GEMM."""

    @staticmethod
    def forward(ctx, x, kernel, stride, padding, dilation):
        x = _f32(x).contiguous()
        B, C, H, W = x.shape
        (kh, kw), (sh, sw), (ph, pw), (dh, dw) = kernel, stride, padding, dilation
        Ho, Wo = conv_out_size(H, kh, sh, ph, dh), conv_out_size(W, kw, sw, pw, dw)
        K = C * kh * kw
        cols = torch.empty((B * Ho * Wo, K), device=x.device, dtype=torch.float32)
        ctx.geom = (B, C, H, W, kh, kw, Ho, Wo, sh, sw, ph, pw, dh, dw)
        _lib.check(_lib.cuda().fb_im2col(x.data_ptr(), cols.data_ptr(), *ctx.geom, K, _dt(cols), _stream()),
                   "fb_im2col")
        return cols

    @staticmethod
    def backward(ctx, g):
        g = _f32(g).contiguous()
        B, C, H, W = ctx.geom[:4]
        dx = torch.empty((B, C, H, W), device=g.device, dtype=torch.float32)
        _lib.check(_lib.cuda().fb_col2im(g.data_ptr(), dx.data_ptr(), *ctx.geom, g.shape[1], _stream()), "fb_col2im")
        return dx, None, None, None, None


def conv_igemm_ok(x: torch.Tensor, stride, dilation, padding, kernel, groups: int) -> bool:
    """True when ``conv2d`` can take the implicit-GEMM path: CUDA, bf16 autocast on, one group, and either stride 1
    with a data gradient whose padding ``dilation * (kernel - 1) - padding`` is not negative, or any stride without
    dilation (space-to-depth form)."""
    if not (_native(x) and x.dim() == 4 and config.low_precision_active() and groups == 1):
        return False
    if tuple(stride) == (1, 1):
        return (dilation[0] * (kernel[0] - 1) - padding[0] >= 0 and dilation[1] * (kernel[1] - 1) - padding[1] >= 0)
    return tuple(dilation) == (1, 1) and padding[0] >= 0 and padding[1] >= 0


def conv2d_igemm(x, weight, bias, padding=(0, 0), dilation=(1, 1), stride=(1, 1), add=None, act=None):
    """``act(conv(x))`` or ``conv(x) + add`` as one node (csrc/native/conv.cpp) where :func:`conv_igemm_ok` says so.  All
    three products read NHWC bf16 activations through 4-D TMA boxes shifted by the filter tap (no window matrix); strides
    are gone after a space-to-depth layout.  ``act``: None or "relu".  Counterpart of the reference's direct loops
    (ferrum-nn/src/conv.rs:209-330)."""
    return _lib.native().conv2d(x, weight, bias, add, stride, padding, dilation, _gemm.ACT[act])


def conv_block(x, w1, w2, down, geometry):
    """A residual block as one node (csrc/native/conv.cpp); ``geometry``: (stride, padding, dilation) of each convolution."""
    g = [[list(v) for v in three] for three in geometry]
    return _lib.native().conv_block(x, w1, w2, down, g[0], g[1], g[2] if down is not None else [])


def im2col(x, kernel, stride=(1, 1), padding=(0, 0), dilation=(1, 1)):
    """Window matrix of a convolution with rows ordered (b, oh, ow) and columns (c, ki, kj)."""
    if _native(x):
        return _Im2colFn.apply(x, tuple(kernel), tuple(stride), tuple(padding), tuple(dilation))
    cols = torch.nn.functional.unfold(x, kernel, dilation=dilation, padding=padding, stride=stride)
    return cols.transpose(1, 2).reshape(-1, cols.shape[1])


class _Pool2dFn(Function):
    @staticmethod
    def forward(ctx, x, kernel, stride, op):
        x = _f32(x).contiguous()
        B, C, H, W = x.shape
        (kh, kw), (sh, sw) = kernel, stride
        Ho, Wo = (H - kh) // sh + 1, (W - kw) // sw + 1
        y = torch.empty((B, C, Ho, Wo), device=x.device, dtype=torch.float32)
        arg = torch.empty((B, C, Ho, Wo), device=x.device, dtype=torch.int32) if op == 0 else None
        ctx.geom, ctx.op = (B, C, H, W, kh, kw, Ho, Wo, sh, sw), op
        _lib.check(_lib.cuda().fb_pool2d_fwd(x.data_ptr(), y.data_ptr(), arg.data_ptr() if arg is not None else None,
                                             *ctx.geom, op, _stream()), "fb_pool2d_fwd")
        ctx.save_for_backward(arg) if arg is not None else None
        return y

    @staticmethod
    def backward(ctx, g):
        g = _f32(g).contiguous()
        arg = ctx.saved_tensors[0] if ctx.op == 0 else None
        B, C, H, W = ctx.geom[:4]
        dx = torch.empty((B, C, H, W), device=g.device, dtype=torch.float32)
        _lib.check(_lib.cuda().fb_pool2d_bwd(g.data_ptr(), arg.data_ptr() if arg is not None else None, dx.data_ptr(),
                                             *ctx.geom, ctx.op, _stream()), "fb_pool2d_bwd")
        return dx, None, None, None


def pool2d(x, kernel, stride, op: str):
    """Max / average pooling over unpadded windows (ferrum-nn/src/conv.rs:340-441)."""
    if _native(x) and x.dim() == 4:
        return _Pool2dFn.apply(x, tuple(kernel), tuple(stride), 0 if op == "max" else 1)
    fn = torch.nn.functional.max_pool2d if op == "max" else torch.nn.functional.avg_pool2d
    return fn(x, kernel, stride)
