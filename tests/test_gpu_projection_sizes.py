"""The tensor-core projections at sizes that are no multiple of their tiles (128 weight rows, 32 and 16 floats of K,
64 complex columns), odd lengths and padded rows, against float64.  Bound: the products are rounded to about
2^-21 each, the sums to 2^-23 of a chain of 32; 1e-6 of the largest output is a few times what both give."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _cn(g, *shape):
    return torch.complex(torch.randn(*shape, generator=g), torch.randn(*shape, generator=g)).cuda()


def _close(got, want):
    from lrnnx_b200 import _lib
    torch.cuda.synchronize()
    assert _lib.lib().b200_device_status() == 0
    assert got.shape == want.shape
    assert float((got.to(torch.complex128) - want).abs().max()) <= 1e-6 * float(want.abs().max())


@pytest.mark.parametrize("M,K,N", [(32, 32, 1), (33, 47, 63), (128, 49, 64), (129, 32, 65), (200, 130, 257), (256, 512, 129)])
@pytest.mark.parametrize("conj", [False, True])
def test_product(M, K, N, conj):
    from lrnnx_b200.ops import projection
    g = torch.Generator().manual_seed(M + K + N)
    W, x = _cn(g, *((K, M) if conj else (M, K))), _cn(g, 3, K, N)
    want = torch.einsum("mk,bkn->bmn", (W.mH if conj else W).to(torch.complex128), x.to(torch.complex128))
    assert projection.fits(W.mH if conj else W, x)
    _close(projection.product(W, x, conj), want)
    padded = projection.product(W, x, conj, padded=True)
    assert padded.stride(1) % 2 == 0
    _close(padded, want)
    _close(projection.product(W.conj().resolve_conj(), torch.cat([x, x], 2)[..., :N], conj).conj(),
           torch.einsum("mk,bkn->bmn", (W.mH if conj else W).to(torch.complex128), x.conj().to(torch.complex128)))


@pytest.mark.parametrize("M,N,L", [(32, 33, 1), (40, 129, 7), (128, 128, 9), (130, 64, 255), (257, 200, 1999)])
def test_gradient(M, N, L):
    from lrnnx_b200.ops import projection
    g = torch.Generator().manual_seed(M + N + L)
    a, b = _cn(g, 3, M, L), _cn(g, 3, N, L)
    want = torch.einsum("bml,bnl->mn", a.to(torch.complex128), b.to(torch.complex128).conj())
    assert projection.grad_fits(a, b)
    _close(projection.gradient(a, b), want)
    _close(projection.gradient(projection.rows(a), projection.rows(b)), want)


@pytest.mark.parametrize("L", [63, 64, 2049])
def test_simplified_scan_at_odd_lengths(L):
    """Intermediate results in padded rows: output and gradients agree with the einsum formulation on the same scan kernels."""
    from lrnnx_b200.ops import simplified_scan_fn
    from oracle import scan_oracle as O
    g = torch.Generator().manual_seed(L)
    P, H = 48, 40
    A = torch.complex(-0.05 - 0.1 * torch.rand(P, generator=g), torch.rand(P, generator=g))
    t = [_cn(g, 2, H, L).cpu(), 0.5 + torch.rand(2, P, L, generator=g), A, _cn(g, P, H).cpu() / H ** 0.5, _cn(g, H, P).cpu() / P ** 0.5]
    gout = _cn(g, 2, H, L).cpu()

    def run(fn, cast, **kw):
        leaves = [cast(v).requires_grad_(True) for v in t]
        y = fn(*leaves, discretization="zoh", **kw)
        return [y.detach().cpu()] + [v.cpu() for v in torch.autograd.grad(y, leaves, cast(gout))]

    wide = lambda v: v.to(torch.complex128 if v.is_complex() else torch.float64)  # noqa: E731
    want = run(O.simplified_scan_oracle, wide, compute_dtype=torch.float64)
    for a, b in zip(run(simplified_scan_fn, lambda v: v.cuda()), want):
        assert float((wide(a) - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.parametrize("L", [63, 64])
def test_the_extension_lays_its_outputs_out_as_before(L):
    """A caller's own view of rows that are one element longer gets dense outputs, as any other input; padded rows are for
    callers that ask for them."""
    from lrnnx_b200 import simplified_scan_cuda as ext
    g = torch.Generator().manual_seed(L)
    u, dout = _cn(g, 2, 40, L + 1)[..., :L], _cn(g, 2, 40, L + 1)[..., :L]
    delta, A, one = torch.ones(2, 40, L, device="cuda"), -torch.rand(40, 1, device="cuda").to(torch.complex64), torch.ones(40, 1, device="cuda", dtype=torch.complex64)
    for kw, pitch in (({}, L), ({"padded": True}, L + L % 2)):
        out, x = ext.fwd(u, delta, A, one, one, None, "zoh", **kw)
        du = ext.bwd(u, delta, A, one, one, None, dout, x, "zoh", **kw)[0]
        assert out.stride() == du.stride() == (40 * pitch, pitch, 1)


def _plain(spec, a, b):
    """The complex sum as four real ones in float64: what is infinite or not a number follows from IEEE arithmetic alone."""
    a, b = a.cpu().to(torch.complex128), b.cpu().to(torch.complex128)
    e = lambda x, y: torch.einsum(spec, x, y)  # noqa: E731
    return e(a.real, b.real) - e(a.imag, b.imag), e(a.real, b.imag) + e(a.imag, b.real)


def _same_specials(got, want):
    for x, y in zip((got.real.cpu().double(), got.imag.cpu().double()), want):
        assert torch.equal(x.isnan(), y.isnan())
        fin = y.isfinite()
        assert torch.equal(x[~fin & ~y.isnan()], y[~fin & ~y.isnan()])          # infinities and their signs
        assert bool(fin.any())
        assert float((x - y)[fin].abs().max()) <= 1e-6 * float(y[fin].abs().max())


@pytest.mark.parametrize("M,K,N", [(40, 47, 77), (130, 64, 129), (256, 128, 192)])
def test_infinities_and_nans(M, K, N):
    """An infinite or missing value in either operand reaches the outputs that depend on it, as in any float32 product, and
    no others; a weight that is zero or exact in TF32 makes no NaN of an infinity; the largest float32 stays finite."""
    from lrnnx_b200.ops import projection
    g = torch.Generator().manual_seed(M)
    inf, nan = float("inf"), (torch.zeros(1, device="cuda") / torch.zeros(1, device="cuda"))[0]       # the device's own NaN
    W, x = _cn(g, M, K), _cn(g, 2, K, N)
    W[:, 3] = 0.5 + 0.25j                                       # exact in TF32: their low parts are 0
    x[0, 3, 5], x[1, 7, N - 1], x[0, 9, 20] = complex(inf, 0), complex(2, -inf), complex(nan, 1)
    _same_specials(projection.product(W, x), _plain("mk,bkn->bmn", W, x))
    _same_specials(projection.product(W.mH.contiguous(), x, True), _plain("mk,bkn->bmn", W, x))
    W[11, 0], W[M - 1, 2], W[20, K - 1] = complex(inf, 1), complex(0.5, nan), 3.4028e38
    x = 1e-30 * _cn(g, 2, K, N)
    _same_specials(projection.product(W, x), _plain("mk,bkn->bmn", W, x))

    a, b = _cn(g, 2, M, N), _cn(g, 2, K, N)
    b[:, 1] = 1 + 0.5j
    a[0, 3, 5], a[1, M - 1, N - 1], b[1, K - 1, 0] = complex(inf, 0), complex(1, nan), complex(0, -inf)
    _same_specials(projection.gradient(a, b), _plain("bml,bnl->mn", a, b.conj()))


def _errors(got, want):
    """(2-norm of the error over that of the result, the error's share along the result)"""
    e = got.to(torch.complex128) - want
    return float(e.norm() / want.norm()), float((want.conj() * e).sum().real / want.norm() ** 2)


@pytest.mark.parametrize("real", [True, False])
@pytest.mark.parametrize("K", [64, 80, 95, 96, 130, 384, 1000])
def test_error_against_a_float32_product(K, real):
    """The error is no larger than a float32 einsum's, and not to one side (an error to one side adds up over the scan
    behind it; truncation in the accumulator alone would make 1.3e-7)."""
    from lrnnx_b200.ops import projection
    g = torch.Generator().manual_seed(K)
    W, x = _cn(g, 100, K), _cn(g, 2, K, 2001)
    if real:
        x = torch.complex(x.real, torch.zeros_like(x.real))
    want = torch.einsum("mk,bkn->bmn", W.to(torch.complex128), x.to(torch.complex128))
    err, side = _errors(projection.product(W, x), want)
    err32, _ = _errors(torch.einsum("mk,bkn->bmn", W, x), want)
    assert err <= 1.02 * err32 and abs(side) <= 3e-8, (err, err32, side)


@pytest.mark.parametrize("real", [True, False])
@pytest.mark.parametrize("batch,L", [(1, 1024), (2, 1999)])
def test_error_of_the_gradient_against_a_float32_product(batch, L, real):
    from lrnnx_b200.ops import projection
    g = torch.Generator().manual_seed(L)
    a, b = _cn(g, batch, 100, L), _cn(g, batch, 50, L)
    if real:
        b = torch.complex(b.real, torch.zeros_like(b.real))
    want = torch.einsum("bml,bnl->mn", a.to(torch.complex128), b.to(torch.complex128).conj())
    err, side = _errors(projection.gradient(a, b), want)
    err32, _ = _errors(torch.einsum("bml,bnl->mn", a, b.conj()), want)
    assert err <= 1.02 * err32 and abs(side) <= 3e-8, (err, err32, side)


@pytest.mark.parametrize("P,H,L,disc", [(192, 112, 81, "zoh"), (176, 328, 64, "dirac"), (56, 400, 515, "bilinear")])
def test_simplified_scan_is_as_exact_as_with_einsums(P, H, L, disc, monkeypatch):
    """The whole op against float64: an error of the products to one side would add up over the scan, and to the scan's
    own (5 to 10 % more than with float32 einsums in place of the kernels)."""
    from lrnnx_b200.ops import projection, simplified_scan_fn
    from oracle import scan_oracle as O
    g = torch.Generator().manual_seed(P)
    r = lambda *s: torch.rand(*s, generator=g)  # noqa: E731
    A = torch.log(torch.polar(0.9 + 0.099 * r(P), torch.pi / 10 * r(P)))
    u = torch.complex(torch.randn(2, H, L, generator=g), torch.zeros(2, H, L))
    t = [u, torch.ones(2, P, L) if disc == "dirac" else 0.5 + r(2, P, L), A, _cn(g, P, H).cpu() / H ** 0.5, _cn(g, H, P).cpu() / P ** 0.5]
    gout = _cn(g, 2, H, L).cpu()

    def run(fn, cast, **kw):
        leaves = [cast(v).requires_grad_(True) for v in t]
        y = fn(*leaves, discretization=disc, **kw)
        return [y.detach().cpu()] + [v.cpu() for v in torch.autograd.grad(y, leaves, cast(gout))]

    wide = lambda v: v.to(torch.complex128 if v.is_complex() else torch.float64)  # noqa: E731
    want = run(O.simplified_scan_oracle, wide, compute_dtype=torch.float64)
    err = lambda: [float((wide(a) - b).norm() / b.norm()) for a, b in zip(run(simplified_scan_fn, lambda v: v.cuda()), want)]  # noqa: E731
    here = err()
    monkeypatch.setattr(projection, "fits", lambda W, x: False)
    monkeypatch.setattr(projection, "grad_fits", lambda g, u: False)
    ratios = [a / b for a, b in zip(here, err())]
    assert sum(ratios) / len(ratios) <= 1.02, ratios
