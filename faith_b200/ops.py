"""Thin tensor-level wrappers over the C ABI: argument checks, output allocation, stream.

PyTorch is used only for device memory and the current stream; all arithmetic happens in
libfaith_b200.so.  Every tensor must be a contiguous float32 CUDA tensor.  The operators of the `Bounds` class go through
the native boundary (csrc/binding/binding.cpp): their small calls are bound by the host, and the same steps over ctypes cost 25
to 40 us per operator; the remaining entry points, which the C++ driver calls itself, are bound here with ctypes.
"""
import math

import torch

from . import _lib
from ._lib import (FB_EXP, FB_NATIVE, FB_P1, FB_P2, FB_PINF, FB_RECIPROCAL, FB_RELU, FB_TANH, FB_TRANSPOSED,
                   check, load)


def norm_code(p):
    """Maps the perturbation norm p to the C enum (the dual exponent is implied)."""
    if p == 1:
        return FB_P1
    if p == 2:
        return FB_P2
    if p == float("inf") or p >= 10:  # the reference treats p >= 10 as infinity (Verifier.py:17)
        return FB_PINF
    raise ValueError("only p in {1, 2, inf} is supported, got %r" % (p,))


def _chk(*tensors):
    dev = None
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda:
            raise _lib.FaithError("faith_b200 operators need CUDA tensors (there is no CPU path)")
        if t.dtype != torch.float32:
            raise _lib.FaithError("float32 tensors required, got %s" % t.dtype)
        if not t.is_contiguous():
            raise _lib.FaithError("contiguous tensors required")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise _lib.FaithError("all tensors must live on one device")
    return dev


_native = _lib.binding


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _p(t):
    return None if t is None else t.data_ptr()


def concretize(lw, uw, lb, ub, p, eps, words=1, layout=FB_NATIVE):
    return _native().concretize(lw, uw, lb, ub, p, eps, words, layout)


def relax(op, lw, uw, lb, ub, p, eps, words=1, layout=FB_NATIVE, out=None, violation=None):
    return _native().relax(op, lw, uw, lb, ub, p, eps, words, layout, out, violation)


def relax_checked(op, lw, uw, lb, ub, p, eps, words=1):
    """relax() that also reads the status word of the call back (waits for the stream): (lw, uw, lb, ub, word)."""
    return _native().relax_checked(op, lw, uw, lb, ub, p, eps, words)


def matmul(lw, uw, lb, ub, W, bias=None):
    return _native().matmul(lw, uw, lb, ub, W, bias)


def relax_coef(op, lw, uw, lb, ub, p, eps, words=1, violation=None):
    """Relaxation without the rescale pass: returns (c_l, c_u, out_lb, out_ub), all [rows..., Do]."""
    dev = _chk(lw, uw, lb, ub)
    rows = lb.numel() // lb.shape[-1]
    Di, Do = lw.shape[-2], lw.shape[-1]
    out = tuple(torch.empty_like(lb) for _ in range(4))
    with torch.cuda.device(dev):
        check(load().fb_relax_coef_f32(int(op), _p(lw), _p(uw), _p(lb), _p(ub), *[_p(t) for t in out], rows, Di, Do,
                                       int(words), norm_code(p), float(eps), _p(violation), _stream()), "fb_relax_coef_f32")
    return out


def matmul_residual(lw, uw, lb, ub, W, bias, residual, c_l=None, c_u=None):
    """matmul of (lw, uw, lb, ub) (or of (c_l * lw, c_u * uw, lb, ub)) with W, + bias, + residual (lw, uw, lb, ub)."""
    dev = _chk(lw, uw, lb, ub, W, bias, *residual)
    rows = lb.numel() // lb.shape[-1]
    Di, Do = lw.shape[-2], lw.shape[-1]
    Dy = W.shape[0]
    y_lw = torch.empty(lw.shape[:-1] + (Dy,), device=dev, dtype=torch.float32)
    y_uw = torch.empty_like(y_lw)
    y_lb = torch.empty(lb.shape[:-1] + (Dy,), device=dev, dtype=torch.float32)
    y_ub = torch.empty_like(y_lb)
    with torch.cuda.device(dev):
        check(load().fb_matmul_residual_f32(_p(lw), _p(uw), _p(lb), _p(ub), _p(c_l), _p(c_u), _p(W), _p(bias),
                                            *[_p(t) for t in residual], _p(y_lw), _p(y_uw), _p(y_lb), _p(y_ub), rows, Di, Do,
                                            Dy, _stream()), "fb_matmul_residual_f32")
    return y_lw, y_uw, y_lb, y_ub


def row_sums(lw, uw, lb, ub):
    """Row sums of a bound in the form fb_matmul_residual_ln_f32 reads: [2 lines, 4 partial sums, rows * (Di + 1)], the
    whole sum in the first partial sum (weight rows first, then the bias rows)."""
    D = lw.shape[-1]
    out = torch.zeros(2, 4, lw.numel() // D + lb.numel() // D, device=lw.device, dtype=torch.float32)
    out[0, 0] = torch.cat([lw.reshape(-1, D).sum(-1), lb.reshape(-1, D).sum(-1)])
    out[1, 0] = torch.cat([uw.reshape(-1, D).sum(-1), ub.reshape(-1, D).sum(-1)])
    return out


def matmul_residual_ln(lw, uw, lb, ub, W, bias, residual, residual_rowsum, gamma, beta, c_l=None, c_u=None):
    """layer_norm(matmul(x, W) + bias + residual), mode no_var, in one launch.  Returns (z_lw, z_uw, z_lb, z_ub,
    z_rowsum); residual_rowsum / z_rowsum as row_sums() lays them out."""
    dev = _chk(lw, uw, lb, ub, W, bias, *residual, residual_rowsum, gamma, beta)
    rows = lb.numel() // lb.shape[-1]
    Di, Do = lw.shape[-2], lw.shape[-1]
    Dy = W.shape[0]
    z_lw = torch.empty(lw.shape[:-1] + (Dy,), device=dev, dtype=torch.float32)
    z_uw = torch.empty_like(z_lw)
    z_lb = torch.empty(lb.shape[:-1] + (Dy,), device=dev, dtype=torch.float32)
    z_ub = torch.empty_like(z_lb)
    z_rs = torch.empty(2, 4, rows * (Di + 1), device=dev, dtype=torch.float32)
    with torch.cuda.device(dev):
        check(load().fb_matmul_residual_ln_f32(_p(lw), _p(uw), _p(lb), _p(ub), _p(c_l), _p(c_u), _p(W), _p(bias),
                                               *[_p(t) for t in residual], _p(residual_rowsum), _p(gamma), _p(beta),
                                               _p(z_lw), _p(z_uw), _p(z_lb), _p(z_ub), _p(z_rs), rows, Di, Do, Dy, _stream()),
              "fb_matmul_residual_ln_f32")
    return z_lw, z_uw, z_lb, z_ub, z_rs


def relax_coef_given(op, lb, ub, l, u, violation=None):
    """relax_coef for a bound whose concretised range (l, u) is already known: no pass over lw / uw."""
    dev = _chk(lb, ub, l, u)
    rows = lb.numel() // lb.shape[-1]
    out = tuple(torch.empty_like(lb) for _ in range(4))
    with torch.cuda.device(dev):
        check(load().fb_relax_coef_given_f32(int(op), _p(lb), _p(ub), _p(l), _p(u), *[_p(t) for t in out], rows,
                                             lb.shape[-1], _p(violation), _stream()), "fb_relax_coef_given_f32")
    return out


def matmul_coef(lw, uw, lb, ub, c_l, c_u, W, bias=None):
    """matmul of (c_l * lw, c_u * uw, lb, ub) with W (+ bias): the consumer side of relax_coef."""
    dev = _chk(lw, uw, lb, ub, c_l, c_u, W, bias)
    rows = lb.numel() // lb.shape[-1]
    Di, Do = lw.shape[-2], lw.shape[-1]
    Dy = W.shape[0]
    y_lw = torch.empty(lw.shape[:-1] + (Dy,), device=dev, dtype=torch.float32)
    y_uw = torch.empty_like(y_lw)
    y_lb = torch.empty(lb.shape[:-1] + (Dy,), device=dev, dtype=torch.float32)
    y_ub = torch.empty_like(y_lb)
    with torch.cuda.device(dev):
        check(load().fb_matmul_coef_f32(_p(lw), _p(uw), _p(lb), _p(ub), _p(c_l), _p(c_u), _p(W), _p(bias), _p(y_lw), _p(y_uw),
                                        _p(y_lb), _p(y_ub), rows, Di, Do, Dy, _stream()), "fb_matmul_coef_f32")
    return y_lw, y_uw, y_lb, y_ub


def matmul_heads_ranges(lw, uw, lb, ub, W, bias, heads, p, eps, words=1):
    """Projection with head-split store that also returns the concretised range of its result: lw, uw
    [S, L, Di, Do], lb, ub [S, L, Do] -> (y_lw, y_uw [S*heads, L, Di, d], y_lb, y_ub, y_l, y_u [S*heads, L, d]).
    Raises FaithError (FB_ERR_SHAPE) outside the tensor-core shapes with Di == 128 * words."""
    dev = _chk(lw, uw, lb, ub, W, bias)
    S, L, Di, Do = lw.shape
    Dy = W.shape[0]
    d = Dy // heads
    y_lw = torch.empty((S * heads, L, Di, d), device=dev, dtype=torch.float32)
    y_uw = torch.empty_like(y_lw)
    y_lb, y_ub, y_l, y_u = (torch.empty((S * heads, L, d), device=dev, dtype=torch.float32) for _ in range(4))
    ws = torch.empty(2 * S * L * (words + 1) * Dy, device=dev, dtype=torch.float32)
    with torch.cuda.device(dev):
        check(load().fb_matmul_heads_ranges_f32(_p(lw), _p(uw), _p(lb), _p(ub), _p(W), _p(bias), _p(y_lw), _p(y_uw), _p(y_lb),
                                                _p(y_ub), _p(y_l), _p(y_u), _p(ws), S * L, Di, Do, Dy, L, heads, int(words),
                                                norm_code(p), float(eps), _stream()), "fb_matmul_heads_ranges_f32")
    return y_lw, y_uw, y_lb, y_ub, y_l, y_u


def dot_product(x, y, p, eps, words=1, out_scale=1.0, layout=FB_NATIVE, scratch=None, out=None):
    """x, y: (lw, uw, lb, ub).  Returns (z_lw, z_uw, z_lb, z_ub)."""
    return _native().dot_product(*x, *y, p, eps, words, out_scale, layout, scratch, out)


def context_kmajor(x, v, p, eps, words=1, out_scale=1.0, merge_heads=1):
    """Context product with the values in the projection's own layout: x (lw, uw [B, Lx, Di, K], lb, ub
    [B, Lx, K]), v (lw, uw [B, K, Di, Ly], lb, ub [B, K, Ly]).  Returns z as fb_dot_product_heads_f32 does.
    Raises FaithError (FB_ERR_SHAPE) outside the tensor-core shapes."""
    z = _native().context_kmajor(*x, *v, p, eps, words, out_scale, merge_heads)
    if z is None:
        check(2, "fb_context_heads_f32")
    return z


def context(x, v, p, eps, words=1):
    """Context product of any shape with the values in the projection's own layout (fb_context_f32), or None where the
    shape is not one it takes (a few query rows against large values)."""
    return _native().context(*x, *v, p, eps, words)


def mul_bounds(x, y, p, eps, words=1):
    return _native().mul_bounds(*x, *y, p, eps, words)


def add(x, y):
    return _native().add(*x, *y)


def scale(x, c):
    return _native().scale(*x, c)


def mul_features(x, w):
    """x * w with w a vector over the feature axis, split by sign (Bounds.py:653-664)."""
    return _native().mul_features(*x, w)


def interval_mul(xl, xu, yl, yu):
    """Elementwise product of two boxes (Bounds.py:667-678)."""
    dev = _chk(xl, xu, yl, yu)
    zl, zu = torch.empty_like(xl), torch.empty_like(xu)
    with torch.cuda.device(dev):
        check(load().fb_interval_mul_f32(_p(xl), _p(xu), _p(yl), _p(yu), _p(zl), _p(zu), xl.numel(), _stream()),
              "fb_interval_mul_f32")
    return zl, zu


def interval_dot(xl, xu, yl, yu):
    """z[b,i,j] = sum_k [x[b,i,k]] * [y[b,j,k]] for boxes x [B,Lx,K], y [B,Ly,K] (Bounds.py:711-721)."""
    dev = _chk(xl, xu, yl, yu)
    B, Lx, K = xl.shape
    Ly = yl.shape[1]
    if yl.shape[0] != B or yl.shape[2] != K:
        raise _lib.FaithError("interval_dot: shapes %s and %s do not match" % (tuple(xl.shape), tuple(yl.shape)))
    zl = torch.empty(B, Lx, Ly, device=dev, dtype=torch.float32)
    zu = torch.empty_like(zl)
    with torch.cuda.device(dev):
        check(load().fb_interval_dot_f32(_p(xl), _p(xu), _p(yl), _p(yu), _p(zl), _p(zu), B, Lx, Ly, K, _stream()),
              "fb_interval_dot_f32")
    return zl, zu


def rowsum(x):
    return _native().rowsum(*x)


def layernorm_novar(x, gamma, beta, residual=None):
    return _native().layernorm_novar(*x, gamma, beta, residual)


def layernorm_standard_checked(x, gamma, beta, p, eps, words=1):
    """Layer norm with the variance in one kernel (fb_layernorm_standard_f32); waits for the stream and returns
    (lw, uw, lb, ub, status word), or None where the row is too wide for it."""
    return _native().layernorm_standard_checked(*x, gamma, beta, p, eps, words)


def split_heads(x, heads, transpose_ld=False):
    """(lw, uw, lb, ub) [B, L, Di, H*d] -> [B*H, L, Di, d], or [B*H, d, Di, L] with transpose_ld."""
    return _native().split_heads(*x, heads, int(transpose_ld))


def merge_heads(x, heads):
    """(lw, uw, lb, ub) [B*H, L, Di, d] -> [B, L, Di, H*d]."""
    return _native().merge_heads(*x, heads)


def conv2d(x, weight, bias, stride, padding):
    """x: (lw, uw, lb, ub) with lw, uw [B, Di, C, H, W] and lb, ub [B, C, H, W]."""
    return _native().conv2d(*x, weight, bias, stride, padding)


def norm_partials(lw, uw, p):
    """Unfinished dual-norm accumulation of the local dim_in rows: (part_l, part_u), each [.., Do]."""
    dev = _chk(lw, uw)
    Di, Do = lw.shape[-2], lw.shape[-1]
    rows = lw.numel() // (Di * Do)
    shape = lw.shape[:-2] + (Do,)
    part_l, part_u = torch.empty(shape, device=dev), torch.empty(shape, device=dev)
    with torch.cuda.device(dev):
        check(load().fb_norm_partials_f32(_p(lw), _p(uw), _p(part_l), _p(part_u), rows, Di, Do, norm_code(p),
                                          _stream()), "fb_norm_partials_f32")
    return part_l, part_u


def relax_with_norms(op, lw, uw, lb, ub, norm_l, norm_u, p, eps, violation=None):
    dev = _chk(lw, uw, lb, ub, norm_l, norm_u)
    Di, Do = lw.shape[-2], lw.shape[-1]
    rows = lw.numel() // (Di * Do)
    out = (torch.empty_like(lw), torch.empty_like(uw), torch.empty_like(lb), torch.empty_like(ub))
    with torch.cuda.device(dev):
        check(load().fb_relax_with_norms_f32(op, _p(lw), _p(uw), _p(lb), _p(ub), _p(norm_l), _p(norm_u),
                                             *[_p(t) for t in out], rows, Di, Do, norm_code(p), eps,
                                             _p(violation), _stream()), "fb_relax_with_norms_f32")
    return out


def softmax_fused(x, p, eps, words=1, violation=None, ranges=False):
    """Fused softmax bound; returns None when the shape needs the unfused chain.  ranges=True appends the
    concretised range (l, u) of the result to the returned tuple."""
    return _native().softmax(*x, p, eps, words, violation, ranges)


def softmax_checked(x, p, eps, words=1):
    """softmax_fused() that also reads the status word of the call back (waits for the stream): None or
    (lw, uw, lb, ub, word)."""
    return _native().softmax_checked(*x, p, eps, words)