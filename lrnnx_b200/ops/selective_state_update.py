"""``selective_state_update`` on the sm_100a kernel.

Same signature, shape handling and in-place state update as
lrnnx/ops/triton/selective_state_update.py:300-476; arbitrary strides
(including stride-0 broadcasts, the "tied head dim" case of :409-414) and
``state_batch_indices`` are passed through to the kernel.  The call allocates
only ``out`` (through the PyTorch caching allocator, so it is legal inside
``torch.cuda.graph`` capture) and launches on the current stream.
"""
from __future__ import annotations

import functools

import torch

from .. import _lib

_DT = {torch.float32: "B200_F32", torch.float16: "B200_F16", torch.bfloat16: "B200_BF16"}
_METHODS = {"zoh": "B200_DISC_ZOH", "bilinear": "B200_DISC_BILINEAR", "dirac": "B200_DISC_DIRAC",
            "mamba": "B200_DISC_MAMBA", "rglru": "B200_DISC_RGLRU", "s7": "B200_DISC_S7"}


@functools.lru_cache(maxsize=None)
def _codes():
    return {k: _lib.enum(v) for k, v in _DT.items()}, {k: _lib.enum(v) for k, v in _METHODS.items()}


def _dt(t, name):
    if t.dtype not in _DT:
        raise RuntimeError(f"{name} must be float32, float16 or bfloat16")
    return _codes()[0][t.dtype]


def _heads(t, dims, at=1):
    """Shape and strides of t with a heads dimension of 1 at position ``at`` where it has none."""
    shape, stride = tuple(t.shape), t.stride()
    if len(shape) == dims:
        return shape, stride
    if len(shape) != dims - 1:
        raise AssertionError(f"expected {dims - 1} or {dims} dimensions, got {len(shape)}")
    return shape[:at] + (1,) + shape[at:], stride[:at] + (0,) + stride[at:]


def selective_state_update(state, x, dt, A, B, C, D=None, z=None, dt_bias=None, dt_softplus=False, deltaA=None,
                           state_batch_indices=None, discretization="mamba"):
    """state (batch, dim, dstate) or (batch, nheads, dim, dstate), updated in place;
    x, dt, z, deltaA (batch, dim) or (batch, nheads, dim); A (dim, dstate) or (nheads, dim, dstate);
    B, C (batch, dstate) or (batch, ngroups, dstate); D, dt_bias (dim,) or (nheads, dim).
    Returns out with the dtype of x: (batch, nheads, dim) for a state with heads, (batch, dim) otherwise."""
    has_heads = state.dim() > 3
    (_, nheads, dim, dstate), s_state = _heads(state, 4)
    x_shape, s_x = _heads(x, 3)
    dt_shape, s_dt = _heads(dt, 3)
    A_shape, s_A = _heads(A, 3, 0)
    B_shape, s_B = _heads(B, 3)
    C_shape, s_C = _heads(C, 3)
    batch = x_shape[0]
    assert x_shape == (batch, nheads, dim)
    assert dt_shape == x_shape
    assert A_shape == (nheads, dim, dstate)
    ngroups = B_shape[1]
    assert nheads % ngroups == 0, "nheads must be divisible by ngroups"
    assert B_shape == (batch, ngroups, dstate)
    assert C_shape == B_shape
    if D is not None:
        D_shape, s_D = _heads(D, 2, 0)
        assert D_shape == (nheads, dim)
    if z is not None:
        z_shape, s_z = _heads(z, 3)
        assert z_shape == x_shape
    if dt_bias is not None:
        bias_shape, s_bias = _heads(dt_bias, 2, 0)
        assert bias_shape == (nheads, dim)
    if deltaA is not None:
        dA_shape, s_dA = _heads(deltaA, 3)
        assert dA_shape == (batch, nheads, dim)
    if state_batch_indices is not None:
        assert state_batch_indices.shape == (batch,)
        if state_batch_indices.dtype != torch.int32 or not state_batch_indices.is_contiguous():
            raise RuntimeError("state_batch_indices must be a contiguous int32 tensor")
    for name, t in (("state", state), ("x", x), ("dt", dt), ("A", A), ("B", B), ("C", C)):
        if not t.is_cuda:
            raise RuntimeError(f"{name} must be a CUDA tensor")
    if B.dtype != C.dtype:
        raise RuntimeError("B and C must have the same dtype")

    a = _lib.struct("b200_ssu_args")()
    a.batch, a.nheads, a.dim, a.dstate, a.ngroups = batch, nheads, dim, dstate, ngroups
    a.state_dtype, a.x_dtype, a.dt_dtype = _dt(state, "state"), _dt(x, "x"), _dt(dt, "dt")
    a.A_dtype, a.bc_dtype = _dt(A, "A"), _dt(B, "B")
    a.dt_softplus = int(bool(dt_softplus))
    methods = _codes()[1]
    a.method = methods.get(discretization.lower(), methods["mamba"])
    with _lib.on_device(x):
        out = torch.empty_like(x)
        a.state, a.x, a.dt, a.A, a.B, a.C, a.out = (state.data_ptr(), x.data_ptr(), dt.data_ptr(), A.data_ptr(),
                                                    B.data_ptr(), C.data_ptr(), out.data_ptr())
        a.state_bs, a.state_hs, a.state_ds, a.state_ns = s_state
        a.x_bs, a.x_hs, a.x_ds = s_x
        a.dt_bs, a.dt_hs, a.dt_ds = s_dt
        a.A_hs, a.A_ds, a.A_ns = s_A
        a.B_bs, a.B_gs, a.B_ns = s_B
        a.C_bs, a.C_gs, a.C_ns = s_C
        a.out_bs, a.out_hs, a.out_ds = _heads(out, 3)[1]
        if D is not None:
            a.D, a.D_dtype = D.data_ptr(), _dt(D, "D")
            a.D_hs, a.D_ds = s_D
        if z is not None:
            a.z, a.z_dtype = z.data_ptr(), _dt(z, "z")
            a.z_bs, a.z_hs, a.z_ds = s_z
        if dt_bias is not None:
            a.dt_bias, a.dt_bias_dtype = dt_bias.data_ptr(), _dt(dt_bias, "dt_bias")
            a.dt_bias_hs, a.dt_bias_ds = s_bias
        if deltaA is not None:
            a.deltaA, a.deltaA_dtype = deltaA.data_ptr(), _dt(deltaA, "deltaA")
            a.deltaA_bs, a.deltaA_hs, a.deltaA_ds = s_dA
        if state_batch_indices is not None:
            a.state_batch_indices = state_batch_indices.data_ptr()
        _lib.call("b200_ssu_step", a, _lib.stream_of(x))
    if has_heads:
        return out if out.dim() == 3 else out.unsqueeze(1)
    return out if out.dim() == 2 else out.squeeze(1)
