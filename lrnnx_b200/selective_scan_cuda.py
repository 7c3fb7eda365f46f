"""Drop-in for lrnnx's compiled ``selective_scan_cuda`` module.

``fwd`` / ``bwd`` keep the positional signatures bound in
csrc/selective_scan/bindings.cpp:5-8 (declared in
csrc/selective_scan/selective_scan.h:114-136) and reproduce the checks,
allocations and return lists of selective_scan_fwd / selective_scan_bwd
(csrc/selective_scan/selective_scan_cpu.cpp:263-632).  A failed check raises
``RuntimeError`` like the reference's ``TORCH_CHECK``.  Unlike the reference
(selective_scan_cpu.cpp:404,612) fp16 / bf16 activations are accepted; the
recurrence state is always fp32.
"""
from __future__ import annotations

import ctypes
import functools

import torch
from torch.multiprocessing.reductions import StorageWeakRef

from . import _lib

_METHODS = {
    "zoh": "B200_DISC_ZOH",
    "bilinear": "B200_DISC_BILINEAR",
    "dirac": "B200_DISC_DIRAC",
    "mamba": "B200_DISC_MAMBA",
    "s7": "B200_DISC_S7",
    "rglru": "B200_DISC_RGLRU",
}
_DTYPES = {torch.float32: "B200_F32", torch.float16: "B200_F16", torch.bfloat16: "B200_BF16"}
CHUNK = 2048


def _check(cond: bool, msg: str) -> None:
    if not cond:
        raise RuntimeError(msg)


_code = functools.lru_cache(maxsize=None)(_lib.enum)


def _ptr(t):
    return None if t is None else t.data_ptr()


def _shape(t, *shape, name: str) -> None:
    if t.shape != shape:
        raise RuntimeError(f"{name} must have shape {tuple(shape)}, got {tuple(t.shape)}")


def _common(u, delta, A, B, C, D, z, delta_bias, deltaA, discretization):
    """Validation shared by fwd and bwd; returns the partially filled argument block."""
    _check(u.dtype in _DTYPES, "u must be float32, float16 or bfloat16")
    _check(A.dtype in (torch.float32, torch.complex64), "A must be float32 or complex64")
    _check(discretization in _METHODS, "Discretization method not supported")
    is_complex = A.dtype == torch.complex64
    if discretization == "s7":
        _check(not is_complex, "S7 discretization only supports real (float) weights, not complex")
    if discretization == "rglru":
        _check(not is_complex, "RGLRU discretization only supports real (float) weights, not complex")
    var_B, var_C = B.dim() >= 3, C.dim() >= 3
    _check(delta.dtype == u.dtype, "delta must have the dtype of u")
    _check(B.dtype == (u.dtype if var_B else A.dtype), "B has the wrong dtype")
    _check(C.dtype == (u.dtype if var_C else A.dtype), "C has the wrong dtype")
    for name, t in (("u", u), ("delta", delta), ("A", A), ("B", B), ("C", C)):
        if not t.is_cuda:
            raise RuntimeError(f"{name} must be a CUDA tensor")
    _check(u.dim() == 3, "u must be (batch, dim, seqlen)")
    _check(u.stride(-1) == 1 or u.size(-1) == 1, "u must be contiguous in the last dimension")
    _check(delta.stride(-1) == 1 or delta.size(-1) == 1, "delta must be contiguous in the last dimension")
    batch, dim, seqlen = u.shape
    _check(A.dim() == 2, "A must be (dim, dstate)")
    dstate = A.size(1)
    n_groups = B.size(1) if var_B else 1
    _check(dstate <= 256, "selective_scan only supports state dimension <= 256")
    _shape(delta, batch, dim, seqlen, name="delta")
    _shape(A, dim, dstate, name="A")
    lb = seqlen * 2 if is_complex else seqlen
    if var_B:
        _shape(B, batch, n_groups, dstate, lb, name="B")
        _check(B.stride(-1) == 1 or B.size(-1) == 1, "B must be contiguous in the last dimension")
    else:
        _shape(B, dim, dstate, name="B")
    if var_C:
        _shape(C, batch, C.size(1), dstate, lb, name="C")
        _check(C.size(1) == n_groups or not var_B, "B and C must have the same number of groups")
        _check(C.stride(-1) == 1 or C.size(-1) == 1, "C must be contiguous in the last dimension")
        if not var_B:
            n_groups = C.size(1)
    else:
        _shape(C, dim, dstate, name="C")
    _check(dim % n_groups == 0, "dim must be a multiple of the number of groups")
    for name, t in (("D", D), ("delta_bias", delta_bias)):
        if t is not None:
            if t.dtype != torch.float32 or not t.is_cuda or not (t.stride(-1) == 1 or t.size(-1) == 1):
                _check(t.dtype == torch.float32, f"{name} must be float32")
                _check(t.is_cuda, f"{name} must be a CUDA tensor")
                raise RuntimeError(f"{name} must be contiguous")
            _shape(t, dim, name=name)
    for name, t in (("deltaA", deltaA), ("z", z)):
        if t is not None:
            if t.dtype != u.dtype or not t.is_cuda or not (t.stride(-1) == 1 or t.size(-1) == 1):
                _check(t.dtype == u.dtype, f"{name} must have the dtype of u")
                _check(t.is_cuda, f"{name} must be a CUDA tensor")
                raise RuntimeError(f"{name} must be contiguous in the last dimension")
            _shape(t, batch, dim, seqlen, name=name)

    a = _lib.struct("b200_selscan_fwd_args")()
    a.batch, a.dim, a.seqlen, a.dstate, a.n_groups = batch, dim, seqlen, dstate, n_groups
    a.dtype = _code(_DTYPES[u.dtype])
    a.is_complex = int(is_complex)
    a.var_B, a.var_C = int(var_B), int(var_C)
    a.method = _code(_METHODS[discretization])
    a.u, a.delta, a.A, a.B, a.C = u.data_ptr(), delta.data_ptr(), A.data_ptr(), B.data_ptr(), C.data_ptr()
    a.D, a.z, a.delta_bias, a.deltaA = _ptr(D), _ptr(z), _ptr(delta_bias), _ptr(deltaA)
    a.u_bs, a.u_ds, _ = u.stride()
    a.delta_bs, a.delta_ds, _ = delta.stride()
    if z is not None:
        a.z_bs, a.z_ds, _ = z.stride()
    if deltaA is not None:
        a.deltaA_bs, a.deltaA_ds, _ = deltaA.stride()
    a.A_ds, a.A_ns = A.stride()
    if var_B:
        a.B_bs, a.B_gs, a.B_ns, _ = B.stride()
    else:
        a.B_gs, a.B_ns = B.stride()
    if var_C:
        a.C_bs, a.C_gs, a.C_ns, _ = C.stride()
    else:
        a.C_gs, a.C_ns = C.stride()
    return a, (batch, dim, seqlen, dstate, n_groups, is_complex, var_B, var_C)


_stream = _lib.stream_of
_SM_COUNT = {}


def _segments_for(u, batch, dim, seqlen, dstate, n_groups, is_complex, var_B, var_C, deltaA, method, rows=()):
    """Number of sequence segments for the forward call: > 1 only for long rows that would leave
    part of the GPU idle, on the shape class of the state-parallel kernels.  Segments are scanned
    concurrently from zero states and stitched by the summary fold + fix-up that the multi-GPU
    sequence-parallel path uses.  ``rows``: the call's (batch, ..., L) operands."""
    if is_complex or method != "mamba" or not (var_B and var_C) or deltaA is not None or dstate != 16:
        return 1
    if seqlen < 4 * CHUNK:
        return 1
    sms = _sm_count(u)
    if u.dtype != torch.float32:
        # 16-bit outputs behind a cut are rounded twice, by the segment and by the fix-up: the places of the cuts show
        # in the results, and calls without cuts are the more exact.  So only what has always been cut is (whole
        # tiles of 16 channels and 8 steps, in whole 16-byte pieces of rows), and where it has always been.
        return _segments_16bit(batch * dim // 16, seqlen, 8 * sms) if _whole_tiles(dim // n_groups, seqlen, rows) else 1
    blocks = _blocks(batch, dim, n_groups)
    if blocks >= 12 * sms:
        return 1
    best, best_ns = 1, None
    for S, seg_len in _cuts(seqlen):
        ns = _stitched_ns(blocks, S, seg_len, batch * dim, sms)
        if best_ns is None or ns < 0.95 * best_ns:
            best, best_ns = S, ns
    return best


def _blocks(batch, dim, n_groups):
    """Thread blocks of 32 channels, or what takes the place of one; 3 fit on an SM."""
    channels = dim // n_groups
    return batch * n_groups * -(-channels // 32) if channels > 16 else -(-batch * n_groups // 2)


def _walk_ns(blocks, steps, sms):
    # measured: a step of a thread block takes 60, 80 and 105 ns with one, two and three of them on an SM
    step_ns = (0, 60, 80, 105)
    full, rest = divmod(blocks, 3 * sms)
    return (full * step_ns[3] + step_ns[-(-rest // sms)]) * steps


def _stitched_ns(blocks, S, seg_len, rows, sms):
    return _walk_ns(blocks * S, seg_len, sms) + 6 * rows * (S - 1)        # measured: the fix-up takes 6 ns per row and segment


def _two_passes(u, batch, dim, seqlen, n_groups, S):
    """(segments, steps per segment) where a forward call that would run in ``S`` segments (1: none) is faster in two
    passes over shorter ones, else None.  The first pass walks the states of all segments but the last, the second
    starts every segment from where the ones before it end: there is nothing to correct afterwards, so outputs are
    rounded once, and segments may be as short as the idle part of the GPU asks for."""
    return _two_passes_for(_blocks(batch, dim, n_groups), batch * dim, seqlen, S, _sm_count(u))


@functools.lru_cache(maxsize=1024)
def _two_passes_for(blocks, rows, seqlen, S, sms):
    if blocks >= 3 * sms or seqlen < 256:
        return None
    seg_len = -(-(-(-seqlen // S)) // CHUNK) * CHUNK if S > 1 else seqlen
    now = 1.12 * _stitched_ns(blocks, S, seg_len, rows, sms)
    if S > 1:       # the last segment is shorter and fills gaps: between the longest walk and whole waves, 1.2 times the full GPU's rate
        now = min(now, 1.12 * (max(_walk_ns(1, seg_len, sms), 1.2 * 105 * blocks * seqlen / (3 * sms)) + 6 * rows * (S - 1)))
    best, best_ns = None, now
    for want in (2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64):
        seg_len = -(-(-(-seqlen // want)) // 32) * 32
        n = -(-seqlen // seg_len)
        if n < 2 or seg_len < 64:
            break
        # measured: the walks of both passes take 1.5 times one pass' step times (and a plain call 1.12 times them), a
        # launch 4.5 us, the state of an earlier segment 0.1 us, a wave of thread blocks 3.6 us to start
        ns = 1.5 * _walk_ns(blocks * n, seg_len, sms) + 4500 + 100 * n + 3600 * -(-blocks * n // (3 * sms))
        if ns < best_ns:
            best, best_ns = (n, seg_len), ns
    return best if best_ns < 0.9 * now - 4000 else None       # the host's share of a second launch


def _sm_count(u):
    idx = u.device.index if u.device.index is not None else torch.cuda.current_device()
    if idx not in _SM_COUNT:
        _SM_COUNT[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    return _SM_COUNT[idx]


def _cuts(seqlen):
    """Segment counts up to 16, and the segments' length: whole checkpoint chunks, two at least."""
    for want in range(1, 17):
        seg_len = -(-(-(-seqlen // want)) // CHUNK) * CHUNK
        if want > 1 and seg_len < 2 * CHUNK:
            return
        yield -(-seqlen // seg_len), seg_len


def _whole_tiles(channels, seqlen, rows):
    return channels % 16 == 0 and seqlen % 8 == 0 and all(
        t is None or (t.data_ptr() % 16 == 0 and all(s % 8 == 0 for s in t.stride()[:-1])) for t in rows)


def _segments_16bit(tiles, seqlen, slots):
    """The segment count whose ``tiles`` (16 channels each) fill whole waves of ``slots`` best; ties: fewer segments."""
    if tiles >= 4 * slots:
        return 1
    best, best_eff = 1, 0.0
    for S, _ in _cuts(seqlen):
        waves = tiles * S / slots
        eff = waves if waves <= 1.0 else waves / -(-waves // 1)
        if eff > best_eff * 1.10 + 1e-9:
            best, best_eff = S, eff
    return best


# Stage states: the state-parallel kernels pass the state at every stage boundary from the forward to
# the backward call (which then skips recomputing them).  They live behind the checkpoints in x's
# own allocation, so the reference's fwd / bwd signatures stay as they are.  bwd() recognises an x
# made by fwd() through a registry of weak references to the storages fwd() allocated (a copy, a
# user-built x or a recycled address never matches) and falls back to recomputation otherwise.
_STAGE_REGISTRY = {}     # storage impl pointer -> (weak reference to the storage, stage length)


def _stage_numel(batch, dim, seqlen, dstate, stage_len):
    return batch * dim * (-(-seqlen // stage_len)) * dstate


def _register_stage_storage(x, stage_len):
    if len(_STAGE_REGISTRY) > 256:
        for key in [k for k, (ref, _) in _STAGE_REGISTRY.items() if ref.expired()]:
            del _STAGE_REGISTRY[key]
    st = x.untyped_storage()
    _STAGE_REGISTRY[st._cdata] = (StorageWeakRef(st), stage_len)


def _stage_states_of(x_, batch, dim, seqlen, dstate):
    """(device address, stage length) of the stage states behind the checkpoints of an x made by
    fwd(), else (None, 0)."""
    if x_ is None or x_.dtype != torch.float32 or x_.storage_offset() != 0 or not x_.is_contiguous():
        return None, 0
    st = x_.untyped_storage()
    entry = _STAGE_REGISTRY.get(st._cdata)
    if entry is None or entry[0].expired():
        return None, 0
    stage_len = entry[1]
    if st.nbytes() != (x_.numel() + _stage_numel(batch, dim, seqlen, dstate, stage_len)) * 4:
        return None, 0
    return x_.data_ptr() + x_.numel() * 4, stage_len


def _stitch_segments(a, x, S, seqlen, u):
    """Fold the zero-start summaries of the segments (one kernel) and run the fix-up kernel on segments >= 1."""
    seg_len = -(-(-(-seqlen // S)) // CHUNK) * CHUNK
    batch, dim, _, two_n = x.shape
    h_in = torch.empty((S, batch, dim, two_n // 2), dtype=torch.float32, device=x.device)
    p_in = torch.empty_like(h_in)
    q = _lib.struct("b200_selscan_fixup_args")()
    a.l_segments = 0
    q.f = a
    q.h_in, q.p_in = h_in.data_ptr(), p_in.data_ptr()
    q.n_segments, q.seg_len = S, seg_len
    _lib.call("b200_selscan_fold", q, _stream(u))
    _lib.call("b200_selscan_fixup", q, _stream(u))


def fwd(u, delta, A, B, C, D_, z_, delta_bias_, deltaA_, delta_softplus, discretization_method_str):
    """Returns ``[out, x]`` or ``[out, x, out_z]`` (selective_scan_cpu.cpp:418-420)."""
    a, (batch, dim, seqlen, dstate, n_groups, is_complex, var_B, var_C) = _common(
        u, delta, A, B, C, D_, z_, delta_bias_, deltaA_, discretization_method_str)
    n_chunks = (seqlen + CHUNK - 1) // CHUNK
    with _lib.on_device(u):
        out = torch.empty_like(delta)
        out_z = torch.empty_like(z_) if z_ is not None else None
        a.delta_softplus = int(bool(delta_softplus))
        a.out, a.out_z = out.data_ptr(), _ptr(out_z)
        a.out_bs, a.out_ds, _ = out.stride()
        if out_z is not None:
            a.out_z_bs, a.out_z_ds, _ = out_z.stride()
        S = _segments_for(u, batch, dim, seqlen, dstate, n_groups, is_complex, var_B, var_C, deltaA_,
                          discretization_method_str, (u, delta, B, C, z_, out, out_z))
        stage_len = _lib.lib().b200_selscan_stage_states(ctypes.byref(a))     # 256 where the state-parallel kernels take the call
        two = _two_passes(u, batch, dim, seqlen, n_groups, S) if stage_len > 0 else None
        if two:
            S, a.seg_len = two
            seg_work = torch.empty((S, batch * dim, dstate + 1), dtype=torch.float32, device=u.device)
            a.seg_work = seg_work.data_ptr()
        elif S > 1:
            stage_len = 0
        x_numel = batch * dim * n_chunks * dstate * 2
        if stage_len > 0:
            flat = torch.empty(x_numel + _stage_numel(batch, dim, seqlen, dstate, stage_len), dtype=A.dtype,
                               device=u.device)
            x = flat[:x_numel].view(batch, dim, n_chunks, dstate * 2)
            _register_stage_storage(x, stage_len)
            a.stage_h = flat.data_ptr() + x_numel * 4
            a.stage_len = stage_len
        else:
            x = torch.empty((batch, dim, n_chunks, dstate * 2), dtype=A.dtype, device=u.device)
        a.x = x.data_ptr()
        if S > 1:
            a.l_segments = S
            try:
                _lib.call("b200_selscan_fwd", a, _stream(u))
            except RuntimeError as e:
                if "l_segments" not in str(e):
                    raise
                S, a.l_segments = 1, 0       # checkpoints that the state-parallel kernels do not take
                _lib.call("b200_selscan_fwd", a, _stream(u))
            if S > 1 and not two:
                _stitch_segments(a, x, S, seqlen, u)
        else:
            _lib.call("b200_selscan_fwd", a, _stream(u))
    return [out, x] if out_z is None else [out, x, out_z]


def _workspace(numel, device):
    """A workspace of up to ``numel`` bytes: a quarter of it, and so on, where there is no memory for it (the call then
    runs in thinner slices), and None where not even a megabyte is left (the kernels that need none take the call)."""
    while numel > 0:
        try:
            return torch.empty(numel, dtype=torch.uint8, device=device)
        except torch.cuda.OutOfMemoryError:
            numel = numel // 4 if numel >= 1 << 22 else 0
    return None


def bwd(u, delta, A, B, C, D_, z_, delta_bias_, deltaA_, dout, x_, out_, dz_, delta_softplus, recompute_out_z,
        discretization_method_str, h_in=None, q_in=None):
    """Returns ``[du, ddelta, dA, dB, dC, dD, ddelta_bias, (ddeltaA), (dz), (out_z)]``
    (selective_scan_cpu.cpp:627-631); dD / ddelta_bias are None when D / delta_bias are.
    Two additions to the reference signature, for a slice of a sequence-parallel scan (real A):
    ``h_in`` (batch, dim, dstate) float32, the state entering the first step, with ``x_`` holding
    the checkpoints corrected for it; ``q_in``, same shape, the gradient with respect to the state
    after the last step."""
    f, (batch, dim, seqlen, dstate, n_groups, is_complex, var_B, var_C) = _common(
        u, delta, A, B, C, D_, z_, delta_bias_, deltaA_, discretization_method_str)
    _check(dout.dtype == u.dtype, "dout must have the dtype of u")
    _check(dout.is_cuda, "dout must be a CUDA tensor")
    _check(dout.stride(-1) == 1 or dout.size(-1) == 1, "dout must be contiguous in the last dimension")
    _shape(dout, batch, dim, seqlen, name="dout")
    has_z = z_ is not None
    n_chunks = (seqlen + CHUNK - 1) // CHUNK
    with _lib.on_device(u):
        out = dz = out_z = None
        if has_z:
            _check(out_ is not None, "out is required when z is given")
            out = out_
            _check(out.dtype == u.dtype and out.is_cuda, "out must be a CUDA tensor with the dtype of u")
            _check(out.stride(-1) == 1 or out.size(-1) == 1, "out must be contiguous in the last dimension")
            _shape(out, batch, dim, seqlen, name="out")
            if dz_ is not None:
                dz = dz_
                _check(dz.dtype == u.dtype and dz.is_cuda, "dz must be a CUDA tensor with the dtype of u")
                _check(dz.stride(-1) == 1 or dz.size(-1) == 1, "dz must be contiguous in the last dimension")
                _shape(dz, batch, dim, seqlen, name="dz")
            else:
                dz = torch.empty_like(z_)
            if recompute_out_z:
                out_z = torch.empty_like(out)
        if n_chunks > 1:
            _check(x_ is not None, "x is required when seqlen > 2048")
        if x_ is not None:
            _check(x_.dtype == A.dtype and x_.is_cuda and x_.is_contiguous(), "x must be a contiguous CUDA tensor in A's dtype")
            _shape(x_, batch, dim, n_chunks, 2 * dstate, name="x")
        du = torch.empty_like(u)
        ddelta = torch.empty_like(delta)
        dA = torch.empty_like(A)
        dB = torch.empty_like(B) if not var_B else torch.empty_like(B, dtype=torch.float32)
        dC = torch.empty_like(C) if not var_C else torch.empty_like(C, dtype=torch.float32)
        dD = torch.empty_like(D_) if D_ is not None else None
        ddelta_bias = torch.empty_like(delta_bias_) if delta_bias_ is not None else None
        # one launch for all the accumulators; each is a tensor of its own, which a caller may keep without the others
        sums = [dA, dB, dC]
        if dD is not None:
            sums.append(dD)
        if ddelta_bias is not None:
            sums.append(ddelta_bias)
        torch._foreach_zero_(sums)
        ddeltaA = torch.empty_like(deltaA_) if deltaA_ is not None else None

        q = _lib.struct("b200_selscan_bwd_args")()
        f.delta_softplus = int(bool(delta_softplus))
        f.x = _ptr(x_)
        f.stage_h, f.stage_len = _stage_states_of(x_, batch, dim, seqlen, dstate)
        f.out = _ptr(out)
        if out is not None:
            f.out_bs, f.out_ds, _ = out.stride()
        f.out_z = _ptr(out_z)
        if out_z is not None:
            f.out_z_bs, f.out_z_ds, _ = out_z.stride()
        q.dout, q.du, q.ddelta = dout.data_ptr(), du.data_ptr(), ddelta.data_ptr()
        q.ddeltaA, q.dz = _ptr(ddeltaA), _ptr(dz)
        q.dA, q.dB, q.dC = dA.data_ptr(), dB.data_ptr(), dC.data_ptr()
        q.dD, q.ddelta_bias = _ptr(dD), _ptr(ddelta_bias)
        if h_in is not None or q_in is not None:
            _check(not is_complex, "h_in / q_in need a real A")
            keep = []
            for name, t in (("h_in", h_in), ("q_in", q_in)):
                if t is None:
                    continue
                _check(t.is_cuda and tuple(t.shape) == (batch, dim, dstate), f"{name} must be a CUDA tensor (batch, dim, dstate)")
                t = t.to(torch.float32).contiguous()
                keep.append(t)
                setattr(q, name, t.data_ptr())
            if h_in is not None:
                f.stage_h, f.stage_len = None, 0      # stage states of a zero-start forward do not apply
        q.dout_bs, q.dout_ds, _ = dout.stride()
        q.du_bs, q.du_ds, _ = du.stride()
        q.ddelta_bs, q.ddelta_ds, _ = ddelta.stride()
        if ddeltaA is not None:
            q.ddeltaA_bs, q.ddeltaA_ds, _ = ddeltaA.stride()
        if dz is not None:
            q.dz_bs, q.dz_ds, _ = dz.stride()
        q.dA_ds, q.dA_ns = dA.stride()
        if var_B:
            q.dB_bs, q.dB_gs, q.dB_ns, _ = dB.stride()
        else:
            q.dB_bs, q.dB_gs, q.dB_ns = 0, dB.stride(0), dB.stride(1)
        if var_C:
            q.dC_bs, q.dC_gs, q.dC_ns, _ = dC.stride()
        else:
            q.dC_bs, q.dC_gs, q.dC_ns = 0, dC.stride(0), dC.stride(1)
        q.f = f
        work = _workspace(_lib.lib().b200_selscan_bwd_work_bytes(ctypes.byref(q)), u.device)
        if work is not None:
            q.work, q.work_bytes = work.data_ptr(), work.numel()
        _lib.call("b200_selscan_bwd", q, _stream(u))
        result = [du, ddelta, dA, dB.to(B.dtype), dC.to(C.dtype), dD, ddelta_bias]
        if deltaA_ is not None:
            result.append(ddeltaA)
        if has_z:
            result.append(dz)
        if recompute_out_z:
            result.append(out_z)
    return result
