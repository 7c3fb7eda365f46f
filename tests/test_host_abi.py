"""CPU-side checks: the C-ABI library loads, exports every symbol the header declares, the
parsed argument-block layouts agree with the compiled ones, and argument validation rejects
bad calls before anything is launched (no compute calls here; no GPU needed)."""
from __future__ import annotations

import ctypes

import pytest
import torch

from lrnnx_b200 import _lib


def test_library_exports_every_declared_symbol():
    lib = _lib.lib()
    structs, enums, functions = _lib.parse_header()
    assert set(functions) == set(_lib.ENTRY_POINTS)
    for fn in functions:
        assert hasattr(lib, fn), f"{fn} declared in include/lrnnx_b200.h but not exported"
    assert lib.b200_abi_version() >= 1


def test_struct_layouts_match_library():
    lib = _lib.lib()
    structs = _lib.parse_header()[0]
    assert len(structs) >= 6
    for name, st in structs.items():
        assert lib.b200_sizeof(name.encode()) == ctypes.sizeof(st), name
    assert lib.b200_sizeof(b"no_such_struct") == -1


def test_enums_follow_reference_order():
    # csrc/selective_scan/selective_scan.h:14-21 and the Triton map at
    # lrnnx/ops/triton/selective_state_update.py:374-382
    assert [_lib.enum(n) for n in ("B200_DISC_ZOH", "B200_DISC_BILINEAR", "B200_DISC_DIRAC", "B200_DISC_MAMBA",
                                   "B200_DISC_RGLRU", "B200_DISC_S7")] == [0, 1, 2, 3, 4, 5]


def test_null_and_range_checks_return_errors_without_launching():
    lib = _lib.lib()
    a = _lib.struct("b200_selscan_fwd_args")()
    assert lib.b200_selscan_fwd(ctypes.byref(a), None) == _lib.enum("B200_ERR_NULL")
    assert b"non-null" in lib.b200_last_error()
    assert lib.b200_selscan_fwd(None, None) == _lib.enum("B200_ERR_NULL")
    buf = (ctypes.c_float * 64)()
    p = ctypes.addressof(buf)
    a.u = a.delta = a.A = a.B = a.C = a.out = a.x = p
    a.batch = a.dim = a.seqlen = a.n_groups = 1
    a.dstate = 300
    assert lib.b200_selscan_fwd(ctypes.byref(a), None) == _lib.enum("B200_ERR_SHAPE")
    assert b"<= 256" in lib.b200_last_error()
    a.dstate, a.method = 4, 17
    assert lib.b200_selscan_fwd(ctypes.byref(a), None) == _lib.enum("B200_ERR_DTYPE")
    a.method, a.is_complex = _lib.enum("B200_DISC_S7"), 1
    assert lib.b200_selscan_fwd(ctypes.byref(a), None) == _lib.enum("B200_ERR_DTYPE")
    s = _lib.struct("b200_simpscan_args")()
    assert lib.b200_simpscan_fwd(ctypes.byref(s), None) == _lib.enum("B200_ERR_NULL")
    q = _lib.struct("b200_s4_args")()
    assert lib.b200_cauchy_bwd(ctypes.byref(q), None) == _lib.enum("B200_ERR_NULL")
    u = _lib.struct("b200_ssu_args")()
    assert lib.b200_ssu_step(ctypes.byref(u), None) == _lib.enum("B200_ERR_NULL")


def test_selscan_bwd_refuses_a_misaligned_workspace():
    """Its boundary states are written 32 bytes at a time."""
    lib = _lib.lib()
    buf = (ctypes.c_float * 4096)()
    p = -(-ctypes.addressof(buf) // 32) * 32
    q = _lib.struct("b200_selscan_bwd_args")()
    f = _lib.struct("b200_selscan_fwd_args")()
    f.batch = f.dim = f.n_groups = f.var_B = f.var_C = 1
    f.seqlen, f.dstate, f.method = 8, 16, _lib.enum("B200_DISC_MAMBA")
    f.u = f.delta = f.A = f.B = f.C = f.out = f.x = p
    f.A_ns, f.B_ns, f.C_ns = 1, 8, 8
    q.f = f
    q.dout = q.du = q.ddelta = q.dA = q.dB = q.dC = p
    q.work_bytes = lib.b200_selscan_bwd_work_bytes(ctypes.byref(q))
    assert q.work_bytes > 0
    q.work = p + 16
    assert lib.b200_selscan_bwd(ctypes.byref(q), None) == _lib.enum("B200_ERR_ALIGN")
    assert b"32-byte" in lib.b200_last_error()


@pytest.mark.parametrize("batch,dim,seqlen,groups", [(8, 1536, 2048, 1), (1, 5120, 131072, 1), (1, 2560, 1 << 20, 1), (2, (1 << 18) + 32, 4096, 1),
                                                     (1, 1 << 20, 100, 1 << 10), (1, 8, 1 << 28, 8)])
def test_selscan_bwd_workspace_is_bounded(batch, dim, seqlen, groups):
    lib = _lib.lib()
    q = _lib.struct("b200_selscan_bwd_args")()
    f = _lib.struct("b200_selscan_fwd_args")()
    f.batch, f.dim, f.n_groups, f.seqlen, f.dstate = batch, dim, groups, seqlen, 16
    f.method, f.var_B, f.var_C = _lib.enum("B200_DISC_MAMBA"), 1, 1
    f.u = f.delta = f.A = f.B = f.C = f.x = 1 << 20
    q.f = f
    assert 0 < lib.b200_selscan_bwd_work_bytes(ctypes.byref(q)) <= 2 << 30


def test_selscan_bwd_workspace_shrinks_without_memory(monkeypatch):
    """The call takes what the allocator has, and goes without where it has nothing."""
    from lrnnx_b200 import selective_scan_cuda as ext
    empty, room = torch.empty, [0]

    def limited(n, **kw):
        if n > room[0]:
            raise torch.cuda.OutOfMemoryError
        return empty(n, dtype=torch.uint8)

    monkeypatch.setattr(torch, "empty", limited)
    for have, got in ((1 << 40, 3 << 28), (1 << 29, 3 << 26), (1 << 22, 3 << 20), (1 << 10, None)):
        room[0] = have
        work = ext._workspace(3 << 28, "cuda")
        assert (None if work is None else work.numel()) == got
    assert ext._workspace(0, "cuda") is None


def test_scratch_size_query():
    lib = _lib.lib()
    assert lib.b200_s4_bwd_scratch_bytes(0, 1, 1) == 0
    small = lib.b200_s4_bwd_scratch_bytes(4, 2, 17)
    assert small == 4 * 2 * 1 * 2 * 8
    assert lib.b200_s4_bwd_scratch_bytes(4, 2, 1 << 18) > small


def test_python_shims_validate_like_the_reference():
    """Host-side checks mirror the reference's TORCH_CHECKs (selective_scan_cpu.cpp:271-378) and
    fire before any device work, so they can be exercised with CPU tensors."""
    from lrnnx_b200 import selective_scan_cuda, simplified_scan_cuda, structured_kernels
    u = torch.randn(1, 2, 8)
    A = -torch.rand(2, 4)
    with pytest.raises(RuntimeError, match="CUDA"):
        selective_scan_cuda.fwd(u, u, A, A, A, None, None, None, None, False, "mamba")
    with pytest.raises(RuntimeError, match="Discretization method not supported"):
        selective_scan_cuda.fwd(u, u, A, A, A, None, None, None, None, False, "euler")
    with pytest.raises(RuntimeError, match="S7 discretization only supports real"):
        selective_scan_cuda.fwd(u, u, A.to(torch.complex64), A.to(torch.complex64), A.to(torch.complex64), None,
                                None, None, None, False, "s7")
    with pytest.raises(RuntimeError, match="dtype"):
        selective_scan_cuda.fwd(u, u.double(), A, A, A, None, None, None, None, False, "mamba")
    with pytest.raises(RuntimeError, match="complex64"):
        simplified_scan_cuda.fwd(u, u, A, A, A, None, "zoh")
    with pytest.raises(RuntimeError, match="CUDA"):
        structured_kernels.cauchy_mult_sym_fwd(torch.randn(2, 4, dtype=torch.complex64),
                                               torch.randn(8, dtype=torch.complex64),
                                               torch.randn(2, 4, dtype=torch.complex64))


def test_projections_leave_operands_of_two_devices_to_torch():
    """torch's einsum refuses them; a kernel would read the other GPU's addresses."""
    from lrnnx_b200.ops import projection

    class Fake:
        is_cuda, dtype = True, torch.complex64

        def __init__(self, device, *shape):
            self.device, self.shape = torch.device(device), torch.Size(shape)

        def dim(self):
            return len(self.shape)

        def numel(self):
            return self.shape.numel()

    W, x, g = Fake("cuda:0", 64, 48), Fake("cuda:0", 2, 48, 99), Fake("cuda:0", 2, 64, 99)
    assert projection.fits(W, x) and projection.grad_fits(g, x)
    x.device = torch.device("cuda:1")
    assert not projection.fits(W, x) and not projection.grad_fits(g, x)
    assert not projection.supported(W, x) and not projection.grad_supported(g, x)


def test_segments_of_two_passes_make_up_the_sequence():
    lib = _lib.lib()
    buf = (ctypes.c_float * 64)()
    a = _lib.struct("b200_selscan_fwd_args")()
    a.u = a.delta = a.A = a.B = a.C = a.out = a.x = a.seg_work = -(-ctypes.addressof(buf) // 16) * 16
    a.batch = a.dim = a.n_groups = a.var_B = a.var_C = 1
    a.seqlen, a.dstate, a.method = 100, 16, _lib.enum("B200_DISC_MAMBA")
    for S, seg_len in ((2, 32), (2, 50), (4, 96), (3, 0), (2, -64), (1 << 20, 1 << 30)):
        a.l_segments, a.seg_len = S, seg_len
        assert lib.b200_selscan_fwd(ctypes.byref(a), None) == _lib.enum("B200_ERR_SHAPE")
    a.l_segments, a.seg_len, a.seg_work = 4, 32, a.seg_work + 4
    assert lib.b200_selscan_fwd(ctypes.byref(a), None) == _lib.enum("B200_ERR_ALIGN")


def test_install_registers_extension_modules():
    import sys
    import lrnnx_b200
    saved = {k: sys.modules.get(k) for k in ("selective_scan_cuda", "simplified_scan_cuda", "structured_kernels")}
    try:
        lrnnx_b200.install()
        import selective_scan_cuda, simplified_scan_cuda, structured_kernels  # noqa: F401
        assert selective_scan_cuda.fwd.__module__ == "lrnnx_b200.selective_scan_cuda"
        assert hasattr(simplified_scan_cuda, "bwd") and hasattr(structured_kernels, "vand_log_mult_sym_bwd")
    finally:
        for k, v in saved.items():
            if v is None:
                sys.modules.pop(k, None)
            else:
                sys.modules[k] = v


def test_every_python_module_of_the_package_imports():
    """Import errors in modules that only the GPU tests use must show up without a GPU."""
    import importlib
    import pkgutil

    import lrnnx_b200
    for mod in pkgutil.walk_packages(lrnnx_b200.__path__, "lrnnx_b200."):
        if mod.name.endswith(".build"):
            continue
        importlib.import_module(mod.name)


def test_16bit_calls_are_cut_where_they_always_were(monkeypatch):
    """16-bit results depend on where a long sequence is cut, because they are rounded once more behind a cut: the cuts of
    whole tiles stay where they were, and other calls stay in one piece."""
    from lrnnx_b200 import selective_scan_cuda as ext
    monkeypatch.setitem(ext._SM_COUNT, 0, 148)

    class U:
        device = torch.device("cuda:0")

    def cuts(dtype, batch, dim, L, groups=1, rows=()):
        U.dtype = dtype
        return ext._segments_for(U, batch, dim, L, 16, groups, False, True, True, None, "mamba", rows)

    for dtype in (torch.bfloat16, torch.float16):
        for shape, want in (((1, 5120, 131072), 7), ((1, 16, 10504), 3), ((1, 512, 32768), 8), ((2, 1024, 16384), 4), ((8, 1536, 16384), 3),
                            ((1, 5120, 8184), 1), ((64, 4096, 8192), 1), ((1, 4096, 65536), 4), ((4, 4736, 32768), 1)):
            assert cuts(dtype, *shape) == want, shape
        assert cuts(dtype, 1, 512, 32767) == cuts(dtype, 1, 520, 32768) == cuts(dtype, 1, 512, 32768, groups=64) == 1
        rows = torch.zeros(1, 8, 40, dtype=dtype)
        assert cuts(dtype, 1, 512, 32768, rows=(rows, None)) == 8
        assert cuts(dtype, 1, 512, 32768, rows=(rows[..., 1:],)) == cuts(dtype, 1, 512, 32768, rows=(rows[..., :39].contiguous(),)) == 1
    assert cuts(torch.float32, 1, 512, 32767) > 1
