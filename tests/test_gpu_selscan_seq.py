"""The state-parallel selective-scan kernels where their tilings can go wrong: channel counts that leave a
warp (8 channels), a thread block (32) or a group partly empty, lengths around the 4-step blocks, the
32-step stages, the 128-step windows, the 256-step pieces and the 2048-step checkpoints, rows that are not
16-byte aligned, orders of the strides, entering states and adjoints, segments of the sequence, and the ways the
backward gets its states and its workspace.  Against the oracle, or against the coverage kernels, which take any
call whose checkpoints are not 16-byte aligned."""
from __future__ import annotations

import pytest
import torch

from conftest import assert_close
from oracle import scan_oracle as O
from test_gpu_selective_scan import ATOL32, GRAD_ATOL32, GRAD_RTOL32, RTOL32, _make_inputs

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8, 1, 1), (2, 3, 3, 1), (1, 33, 31, 1), (2, 40, 32, 2), (1, 24, 33, 3), (2, 72, 127, 1), (1, 16, 129, 2),
          (1, 5, 257, 1), (2, 34, 513, 2), (1, 8, 2047, 1), (1, 9, 2049, 1), (1, 12, 4100, 2)]


def _grads(t, kw, gout, fn):
    leaves = {k: (v.detach().clone().requires_grad_(True) if torch.is_tensor(v) else v) for k, v in t.items()}
    out = fn(**leaves, **kw)
    names = [k for k, v in leaves.items() if torch.is_tensor(v)]
    return out.detach(), dict(zip(names, torch.autograd.grad(out, [leaves[k] for k in names], gout)))


@pytest.mark.parametrize("batch,dim,L,groups", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_edges_of_the_tilings(batch, dim, L, groups, dtype):
    from lrnnx_b200.ops import selective_scan_fn
    t, g = _make_inputs(batch, dim, 16, L, seed=L + dim, dtype=dtype, groups=groups, with_z=L % 2 == 1)
    kw = dict(delta_softplus=True, discretization="mamba")
    gout = torch.randn(batch, dim, L, generator=g).to(dtype)
    out_c, gc = _grads(t, kw, gout, O.selective_scan_oracle)
    out_g, gg = _grads({k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}, kw, gout.cuda(), selective_scan_fn)
    f32 = dtype == torch.float32
    assert_close(out_g.float().cpu(), out_c.float(), rtol=RTOL32 if f32 else 3e-2, atol_scale=ATOL32 if f32 else 1e-2, name="out")
    for k in gc:
        assert_close(gg[k].float().cpu(), gc[k].float(), rtol=GRAD_RTOL32 if f32 else 3e-2, atol_scale=GRAD_ATOL32 if f32 else 2e-2, name=f"d{k}")


@pytest.mark.parametrize("offset", [1, 2, 4])
def test_rows_that_are_not_16_byte_aligned(offset):
    """The same operands as dense tensors and as views that start `offset` elements into wider rows take different
    load paths of the same kernels: outputs are equal bit for bit, gradients up to the order of the atomics."""
    from lrnnx_b200.ops import selective_scan_fn
    t, g = _make_inputs(2, 40, 16, 264, seed=5)
    dense = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    views = dict(dense)
    for k in ("u", "delta", "z", "B", "C"):
        wide = torch.full((*dense[k].shape[:-1], 264 + 9), float("nan"), device="cuda")
        wide[..., offset:offset + 264] = dense[k]
        views[k] = wide[..., offset:offset + 264]
    kw = dict(delta_softplus=True, discretization="mamba")
    gout = torch.randn(2, 40, 264, generator=g).cuda()

    def run(ops):
        leaves = {k: (v.detach().requires_grad_(True) if torch.is_tensor(v) else v) for k, v in ops.items()}
        out = selective_scan_fn(**leaves, **kw)
        return out.detach(), torch.autograd.grad(out, [v for v in leaves.values() if torch.is_tensor(v)], gout)

    (out_a, ga), (out_b, gb) = run(dense), run(views)
    assert torch.equal(out_a, out_b)
    for a, b in zip(ga, gb):
        assert_close(b.cpu(), a.cpu(), rtol=1e-5, atol_scale=1e-6, name="gradient")


@pytest.mark.parametrize("L", [200, 4200])
def test_backward_workspaces(L, monkeypatch):
    """The workspace for the whole batch, for one batch row at a time, and none (the call takes its own): the same
    gradients; and the states rebuilt from the checkpoints alone (an x that did not come from fwd) agree as well."""
    from lrnnx_b200 import _lib
    from lrnnx_b200 import selective_scan_cuda as ext
    t, g = _make_inputs(3, 24, 16, L, seed=L)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    args = (c["u"], c["delta"], c["A"], c["B"], c["C"], c["D"], c["z"], c["delta_bias"], None)
    out, x, _ = ext.fwd(*args, True, "mamba")
    dout = torch.randn(out.shape, generator=g).cuda()
    want = ext.bwd(*args, dout, x, out, None, True, False, "mamba")
    call = _lib.call
    for mode in ("row", "none", "checkpoints"):
        def patched(fn, a, stream, mode=mode):
            if fn == "b200_selscan_bwd" and mode == "row":
                a.work_bytes //= 3
            if fn == "b200_selscan_bwd" and mode == "none":
                a.work = None
            call(fn, a, stream)
        monkeypatch.setattr(_lib, "call", patched)
        got = ext.bwd(*args, dout, x.clone() if mode == "checkpoints" else x, out, None, True, False, "mamba")
        for i, (a, b) in enumerate(zip(got, want)):
            assert_close(a.cpu(), b.cpu(), rtol=2e-5, atol_scale=2e-6, name=f"{mode} gradient {i}")


@pytest.mark.parametrize("stage_len", [512, 1024, 2048, 96])
def test_stage_states_of_another_spacing(stage_len, monkeypatch):
    """A caller of the C entry points that keeps its stage states at a spacing other than the one it was told: the
    backward, which starts walks every 256 steps, recomputes them instead of reading past the ones that are there."""
    from lrnnx_b200 import _lib
    from lrnnx_b200 import selective_scan_cuda as ext
    t, g = _make_inputs(1, 24, 16, 2500, seed=1)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    args = (c["u"], c["delta"], c["A"], c["B"], c["C"], c["D"], c["z"], c["delta_bias"], None)
    out, x, _ = ext.fwd(*args, True, "mamba")
    dout = torch.randn(out.shape, generator=g).cuda()
    want = ext.bwd(*args, dout, x.clone(), out, None, True, False, "mamba")
    room = torch.full((24 * 2500,), float("nan"), device="cuda")       # more than any spacing needs; on both sides of the states
    call = _lib.call

    def patched(fn, a, stream):
        if fn == "b200_selscan_bwd":
            f = a.f
            f.stage_h, f.stage_len = room.data_ptr() + 4 * 16 * 1024, stage_len
            a.f = f
        else:
            a.stage_h, a.stage_len = room.data_ptr() + 4 * 16 * 1024, stage_len
        call(fn, a, stream)

    monkeypatch.setattr(_lib, "call", patched)
    again, x, _ = ext.fwd(*args, True, "mamba")
    assert torch.equal(again, out) and bool(room.isnan().all())
    got = ext.bwd(*args, dout, x.clone(), out, None, True, False, "mamba")
    for i, (a, b) in enumerate(zip(got, want)):
        assert_close(a.cpu(), b.cpu(), rtol=2e-5, atol_scale=2e-6, name=f"gradient {i}")


def test_entering_state_beside_stage_states(monkeypatch):
    """h_in together with the stage states of the zero-start forward, as a caller of the C entry points may hand them
    over: the gradients are those of the entering state."""
    from lrnnx_b200 import _lib
    from lrnnx_b200 import selective_scan_cuda as ext
    t, g = _make_inputs(2, 24, 16, 700, seed=2, with_z=False)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    args = (c["u"], c["delta"], c["A"], c["B"], c["C"], c["D"], None, c["delta_bias"], None)
    out, x = ext.fwd(*args, True, "mamba")
    h_in = torch.randn(2, 24, 16, generator=g).cuda()
    dout = torch.randn(out.shape, generator=g).cuda()
    want = ext.bwd(*args, dout, x, out, None, True, False, "mamba", h_in=h_in)
    ptr, stage_len = ext._stage_states_of(x, 2, 24, 700, 16)
    assert stage_len > 0
    call = _lib.call

    def patched(fn, a, stream):
        f = a.f
        f.stage_h, f.stage_len = ptr, stage_len
        a.f = f
        call(fn, a, stream)

    monkeypatch.setattr(_lib, "call", patched)
    got = ext.bwd(*args, dout, x, out, None, True, False, "mamba", h_in=h_in)
    for i, (a, b) in enumerate(zip(got, want)):
        assert_close(a.cpu(), b.cpu(), rtol=2e-5, atol_scale=2e-6, name=f"gradient {i}")


@pytest.mark.parametrize("dim,groups", [(24, 1), (36, 3), (80, 1)])
@pytest.mark.parametrize("states", ["saved", "checkpoints", "entering"])
def test_slices_of_the_backward(dim, groups, states, monkeypatch):
    """Workspaces that hold a window of the sequence (two and one checkpoint chunks), whole groups, part of a group and a
    single channel, of a length that leaves the last window ragged; with the forward's stage states, with its checkpoints
    alone, and with a state and an adjoint that enter the sequence."""
    from lrnnx_b200 import _lib
    from lrnnx_b200 import selective_scan_cuda as ext
    batch, L = 2, 3 * 2048 + 37
    t, g = _make_inputs(batch, dim, 16, L, seed=dim, groups=groups)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    args = (c["u"], c["delta"], c["A"], c["B"], c["C"], c["D"], c["z"], c["delta_bias"], None)
    out, x, _ = ext.fwd(*args, True, "mamba")
    dout = torch.randn(out.shape, generator=g).cuda()
    kw = {k: torch.randn(batch, dim, 16, generator=g).cuda() for k in ("h_in", "q_in")} if states == "entering" else {}
    if states == "checkpoints":
        x = x.clone()
    call, sizes = _lib.call, []

    def patched(fn, a, stream):
        if fn == "b200_selscan_bwd":
            sizes.append(a.work_bytes)
            a.work_bytes = sizes[-1] if size is None else size
        call(fn, a, stream)

    monkeypatch.setattr(_lib, "call", patched)
    channel = 2048 * 32 + 64
    size = None
    want = ext.bwd(*args, dout, x, out, None, True, False, "mamba", **kw)
    for size in (2 * channel * dim, channel * dim, channel * (dim // groups), channel * 9, channel):
        assert size < sizes[0]
        got = ext.bwd(*args, dout, x, out, None, True, False, "mamba", **kw)
        for i, (a, b) in enumerate(zip(got, want)):
            assert_close(a.cpu(), b.cpu(), rtol=2e-5, atol_scale=2e-6, name=f"{size // channel} channels, gradient {i}")
    size = channel - 1
    with pytest.raises(RuntimeError, match="too small"):
        ext.bwd(*args, dout, x, out, None, True, False, "mamba", **kw)


def test_gradients_own_their_memory():
    """A caller that keeps one gradient keeps that one alone."""
    from lrnnx_b200.ops import selective_scan_fn
    t, g = _make_inputs(2, 24, 16, 40, seed=3)
    kw = dict(delta_softplus=True, discretization="mamba")
    _, grads = _grads({k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}, kw, torch.randn(2, 24, 40, generator=g).cuda(), selective_scan_fn)
    for k, v in grads.items():
        assert v.untyped_storage().nbytes() == v.numel() * v.element_size(), k


def _off_alignment(x):
    """A copy of x that the state-parallel kernels do not take."""
    y = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)[1:].view(x.shape)
    return y.copy_(x)


@pytest.mark.parametrize("batch,dim,groups,L", [(2, 20, 1, 333), (1, 36, 2, 2049), (3, 9, 3, 130)])
@pytest.mark.parametrize("layout", ["dense", "channel-major", "unaligned"])
def test_entering_state_and_adjoint_against_the_coverage_kernels(batch, dim, groups, L, layout):
    from lrnnx_b200 import selective_scan_cuda as ext
    t, g = _make_inputs(batch, dim, 16, L, seed=L, groups=groups)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    dout = torch.randn(batch, dim, L, generator=g).cuda()

    def lay(v):
        if layout == "channel-major":
            return v.transpose(0, 1).contiguous().transpose(0, 1)
        wide = torch.full((*v.shape[:-1], L + 5), float("nan"), device="cuda")
        return wide[..., 3:3 + L].copy_(v) if layout == "unaligned" else v

    for k in ("u", "delta", "z", "B", "C"):
        c[k] = lay(c[k])
    dout = lay(dout)
    args = (c["u"], c["delta"], c["A"], c["B"], c["C"], c["D"], c["z"], c["delta_bias"], None)
    out, x, _ = ext.fwd(*args, True, "mamba")
    for kw in ({}, {"h_in"}, {"q_in"}, {"h_in", "q_in"}):
        kw = {k: torch.randn(batch, dim, 16, generator=g).cuda() for k in sorted(kw)}
        got = ext.bwd(*args, dout, x, out, None, True, False, "mamba", **kw)
        want = ext.bwd(*args, dout, _off_alignment(x), out, None, True, False, "mamba", **kw)
        for i, (a, b) in enumerate(zip(got, want)):
            assert_close(a.cpu(), b.cpu(), rtol=GRAD_RTOL32, atol_scale=GRAD_ATOL32, name=f"{sorted(kw)} gradient {i}")


@pytest.mark.parametrize("dim,groups,L", [(20, 1, 5 * 2048 + 131), (42, 2, 4 * 2048 + 1), (33, 3, 4 * 2048)])
@pytest.mark.parametrize("offset", [0, 1])
def test_segments_at_odd_sizes(dim, groups, L, offset, monkeypatch):
    """A float32 call of few rows is cut into segments at any length, channel count and alignment: outputs, checkpoints
    and gradients against the same call in one piece."""
    from lrnnx_b200 import selective_scan_cuda as ext
    t, g = _make_inputs(1, dim, 16, L, seed=L, groups=groups)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    for k in ("u", "delta", "z", "B", "C"):
        c[k] = torch.full((*c[k].shape[:-1], L + 3), float("nan"), device="cuda")[..., offset:offset + L].copy_(c[k])
    args = (c["u"], c["delta"], c["A"], c["B"], c["C"], c["D"], c["z"], c["delta_bias"], None)
    dout = torch.randn(1, dim, L, generator=g).cuda()
    rule = ext._segments_for
    seen = []

    monkeypatch.setattr(ext, "_two_passes", lambda *a: None)

    def run(S):
        monkeypatch.setattr(ext, "_segments_for", lambda *a: seen.append(rule(*a)) or (seen[-1] if S is None else S))
        out, x, out_z = ext.fwd(*args, True, "mamba")
        return [out, out_z, x] + ext.bwd(*args, dout, x, out, None, True, False, "mamba")

    got, want = run(None), run(1)
    assert seen[0] > 1
    for i, (a, b) in enumerate(zip(got, want)):
        grad = i > 2
        assert_close(a.cpu(), b.cpu(), rtol=GRAD_RTOL32 if grad else RTOL32, atol_scale=GRAD_ATOL32 if grad else ATOL32, name=f"result {i}")


@pytest.mark.parametrize("L", [32, 37, 300])
def test_infinite_decay(L):
    """A state whose A is minus infinity forgets everything at each step, and is no NaN past the end of a ragged sequence.
    (ddelta and dA have the factor A a h, infinity times 0, in them.)"""
    from lrnnx_b200.ops import selective_scan_fn
    t, g = _make_inputs(2, 20, 16, L, seed=L)
    t["A"][:, 3], t["A"][5] = float("-inf"), -3e38
    kw = dict(delta_softplus=True, discretization="mamba")
    gout = torch.randn(2, 20, L, generator=g)
    out_c, gc = _grads(t, kw, gout, O.selective_scan_oracle)
    dev = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    out_g, gg = _grads(dev, kw, gout.cuda(), selective_scan_fn)
    last_c, last_g = (fn(**x, **kw, return_last_state=True)[1] for fn, x in ((O.selective_scan_oracle, t), (selective_scan_fn, dev)))
    for name, a, b in [("out", out_g, out_c), ("last state", last_g, last_c)] + [(k, gg[k], gc[k]) for k in ("u", "B", "C", "D", "z")]:
        assert bool(b.isfinite().all())
        assert_close(a.cpu(), b, rtol=GRAD_RTOL32, atol_scale=GRAD_ATOL32, name=name)


@pytest.mark.parametrize("dim,groups,L", [(20, 1, 700), (33, 3, 2049), (40, 1, 4200), (16, 2, 257)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1])
def test_two_passes(dim, groups, L, dtype, offset, monkeypatch):
    """Segments that start from the states of the ones before them, of one stage, of several and of nearly the whole
    sequence, in aligned and unaligned rows, gated and not: the results of the plain scan (float32 up to the rounding of
    the products that carry a state over a segment), saved states and checkpoints included."""
    from lrnnx_b200 import selective_scan_cuda as ext
    t, g = _make_inputs(2, dim, 16, L, seed=L, dtype=dtype, groups=groups, with_z=L % 2 == 1)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in t.items()}
    for k in ("u", "delta", "B", "C"):
        c[k] = torch.full((*c[k].shape[:-1], L + 3), float("nan"), device="cuda", dtype=dtype)[..., offset:offset + L].copy_(c[k])
    args = (c["u"], c["delta"], c["A"], c["B"], c["C"], c["D"], c["z"], c["delta_bias"], None)
    dout = torch.randn(2, dim, L, generator=g).to(dtype).cuda()
    monkeypatch.setattr(ext, "_segments_for", lambda *a: 1)

    def run(seg_len):
        monkeypatch.setattr(ext, "_two_passes", lambda *a: seg_len and (-(-L // seg_len), seg_len))
        out, x, *rest = ext.fwd(*args, True, "mamba")
        ptr, stage_len = ext._stage_states_of(x, 2, dim, L, 16)
        assert stage_len == 256
        n = 2 * dim * -(-L // 256) * 16
        states = torch.empty(0, dtype=torch.float32, device="cuda").set_(x.untyped_storage(), x.numel(), (n,)).clone()
        grads = ext.bwd(*args, dout, x, out if rest else None, None, True, False, "mamba")
        return [out] + rest, [x, states], grads

    want = run(None)
    f32 = dtype == torch.float32
    for seg_len in (32, 64, 224, (L - 1) // 32 * 32):
        got = run(seg_len)
        # 16-bit outputs are rounded once: they differ where float32 results round apart, by a unit in the last place
        for a, b in zip(got[0], want[0]):
            if not f32:
                assert float((a != b).float().mean()) < 0.02
            assert_close(a.float().cpu(), b.float().cpu(), rtol=1e-5 if f32 else 2 ** -7, atol_scale=2e-6, name=f"{seg_len} output")
        for a, b in zip(got[1], want[1]):
            assert_close(a.cpu(), b.cpu(), rtol=1e-5, atol_scale=2e-6, name=f"{seg_len} states")
        for i, (a, b) in enumerate(zip(got[2], want[2])):
            assert_close(a.float().cpu(), b.float().cpu(), rtol=1e-4 if f32 else 3e-2, atol_scale=1e-5 if f32 else 1e-2, name=f"{seg_len} gradient {i}")


def test_rule_of_the_two_passes():
    """Few rows and a long sequence, at any length, alignment and type; not where the rows fill the GPU."""
    from lrnnx_b200 import selective_scan_cuda as ext
    u = torch.empty(1, device="cuda")
    for batch, dim, L in ((1, 64, 32765), (1, 16, 131072), (2, 512, 16384), (1, 1536, 2048)):
        S, seg_len = ext._two_passes(u, batch, dim, L, 1, 1)
        assert seg_len % 32 == 0 and (S - 1) * seg_len < L <= S * seg_len
    for batch, dim, L in ((8, 1536, 2048), (64, 4096, 512), (1, 64, 200)):
        assert ext._two_passes(u, batch, dim, L, 1, 1) is None
