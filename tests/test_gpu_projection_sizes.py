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
