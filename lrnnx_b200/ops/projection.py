"""Complex projections around the S5 scan on the tensor cores (``b200_cgemm_wx``).

``project(W, x)`` computes ``einsum("mk,bkn->bmn", W, x)`` for complex64 operands, the shape of
Bu = B u, y = C x and of the data gradients du = B^H dBu, dx = C^H dy in lrnnx's
SimplifiedScanFn / S5InnerFn (lrnnx/ops/simplified_scan.py:67,87,136,165,401,419,483-524), with
float32-class accuracy (3xTF32 on tcgen05).  ``project`` and ``weight_grad`` take whole tiles (M a
multiple of 128, K of 32, N of 64; dense, 16-byte aligned x) and reject other shapes.  ``product``
and ``gradient`` take any size: the weight planes are padded, and operands whose rows do not have a pitch
of a multiple of 16 bytes are copied into rows that do (``rows``); the intermediate results of
the S5 wrappers are made that way from the start.
"""
from __future__ import annotations

import torch

from .. import _lib


def _complex_product(W, x) -> bool:
    return (W.is_cuda and W.device == x.device and W.dtype == torch.complex64 and x.dtype == torch.complex64 and W.dim() == 2 and x.dim() == 3
            and x.shape[1] == W.shape[1])


def supported(W, x) -> bool:
    if not _complex_product(W, x):
        return False
    M, K = W.shape
    N = x.shape[2]
    return M % 128 == 0 and K % 32 == 0 and N % 64 == 0 and x.is_contiguous() and x.data_ptr() % 16 == 0


def fits(W, x) -> bool:
    """complex64 operands of a product that fills at least a quarter of the kernel's 128-row weight tile (smaller ones are
    launch latency either way)."""
    return _complex_product(W, x) and min(W.shape) >= 32 and x.numel() > 0


def padded_empty(batch, n, length, like):
    """(batch, n, length) with rows of an even pitch."""
    return torch.empty((batch, n, length + length % 2), dtype=like.dtype, device=like.device)[..., :length]


def _rows_ok(x) -> bool:
    _, n, length = x.shape
    bs, rs, es = x.stride()
    return (es == 1 or length == 1) and rs >= length and rs % 2 == 0 and bs == n * rs and x.data_ptr() % 16 == 0 and not x.is_conj()


def rows(x):
    """x (batch, n, length), or a copy of it, as one run of rows with a 16-byte pitch."""
    if _rows_ok(x):
        return x
    out = padded_empty(*x.shape, x)
    out.copy_(x)
    return out


def weight_planes(W, conj_transpose=False, padded=False):
    """(4, M, K) float32: Re(W) rounded to TF32, the remainder rounded to TF32, and the same for
    Im(W) (one kernel, b200_cgemm_planes).  With ``conj_transpose`` the planes of W^H; with ``padded``
    M and K are the next multiples of 128 and 32, with zeros in the padding."""
    if W.is_conj():
        W = W.resolve_conj()
    n_rows, cols = W.shape
    M, K = (cols, n_rows) if conj_transpose else (n_rows, cols)
    a = _lib.struct("b200_cgemm_planes_args")()
    a.M, a.K, a.conj, a.padded = M, K, int(conj_transpose), int(padded)
    a.w_rs, a.w_cs = (W.stride(1), W.stride(0)) if conj_transpose else (W.stride(0), W.stride(1))
    if padded:
        M, K = -(-M // 128) * 128, -(-K // 32) * 32
    with _lib.on_device(W):
        planes = torch.empty((4, M, K), dtype=torch.float32, device=W.device)
        a.w, a.planes = W.data_ptr(), planes.data_ptr()
        _lib.call("b200_cgemm_planes", a, _lib.stream_of(W))
    return planes


def _wx(W, x, conj_transpose, any_size, padded_out):
    K, M = W.shape if conj_transpose else W.shape[::-1]
    batch, Kx, N = x.shape
    if Kx != K:
        raise RuntimeError(f"project: the weight contracts {K} rows, x has {Kx}")
    planes = weight_planes(W, conj_transpose, any_size)
    a = _lib.struct("b200_cgemm_args")()
    a.batch, a.M, a.K, a.N, a.padded = batch, M, K, N, int(any_size)
    with _lib.on_device(x):
        out = padded_empty(batch, M, N, x) if padded_out else torch.empty((batch, M, N), dtype=torch.complex64, device=x.device)
        a.w_planes, a.x, a.out = planes.data_ptr(), x.data_ptr(), out.data_ptr()
        a.x_bs, a.x_ks, _ = x.stride()
        a.out_bs, a.out_ms, _ = out.stride()
        _lib.call("b200_cgemm_wx", a, _lib.stream_of(x))
    return out


def project(W, x, conj_transpose=False):
    """out[b] = W x[b] (or W^H x[b]): W (M, K) (or (K, M)), x (batch, K, N) -> (batch, M, N), complex64."""
    return _wx(W, x if x.is_contiguous() else x.contiguous(), conj_transpose, False, False)


def product(W, x, conj_transpose=False, padded=False):
    """``project`` for any size; with ``padded`` the rows of the result have an even pitch, as the next
    product wants them."""
    return _wx(W, rows(x), conj_transpose, True, padded)


def grad_supported(g, u) -> bool:
    if not (g.is_cuda and g.device == u.device and g.dtype == torch.complex64 and u.dtype == torch.complex64):
        return False
    if g.dim() != 3 or u.dim() != 3 or g.shape[0] != u.shape[0] or g.shape[2] != u.shape[2]:
        return False
    return g.shape[1] % 128 == 0 and u.shape[1] % 128 == 0 and g.shape[2] % 16 == 0


def grad_fits(g, u) -> bool:
    return (g.is_cuda and g.device == u.device and g.dtype == torch.complex64 and u.dtype == torch.complex64 and g.dim() == 3 and u.dim() == 3
            and g.shape[0] == u.shape[0] and g.shape[2] == u.shape[2] and min(g.shape[1], u.shape[1]) >= 32 and g.numel() > 0)


def _ggh(g, u, any_size):
    a = _lib.struct("b200_cgemm_grad_args")()
    a.batch, a.M, a.L = g.shape
    a.N = u.shape[1]
    with _lib.on_device(g):
        out = torch.zeros((g.shape[1], u.shape[1]), dtype=torch.complex64, device=g.device)
        a.g, a.u, a.out = g.data_ptr(), u.data_ptr(), out.data_ptr()
        if any_size:
            a.g_rs, a.u_rs = g.stride(1), u.stride(1)
        _lib.call("b200_cgemm_grad", a, _lib.stream_of(g))
    return out


def weight_grad(g, u):
    """einsum("bml,bnl->mn", g, conj(u)) for complex64 g (batch, M, L), u (batch, N, L): the
    gradient of a projection weight, summed over batch and time on the tensor cores."""
    return _ggh(g if g.is_contiguous() else g.contiguous(), u if u.is_contiguous() else u.contiguous(), False)


def gradient(g, u):
    """``weight_grad`` for any size."""
    return _ggh(rows(g), rows(u), True)
