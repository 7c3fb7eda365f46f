"""Cauchy kernels at the edges of their tiles: positions go in packed pairs (128 apart in the forward, 256 in the
backward, 512 to a thread block), poles in tiles of 4 and in shared-memory blocks of 1024."""
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _case(rows, n, length):
    g = torch.Generator().manual_seed(rows * 7919 + n * 131 + length)
    r = lambda *s: torch.randn(*s, generator=g)
    v = torch.complex(r(rows, n), r(rows, n))
    w = torch.complex(-0.01 - r(rows, n).abs(), 3 * r(rows, n))
    z = torch.complex(0.05 + 0.05 * r(length).abs(), 4 * r(length))
    return v, z, w, torch.complex(r(rows, length), r(rows, length))


@pytest.mark.parametrize("rows,n,length", [(1, 1, 1), (3, 5, 127), (2, 4, 129), (2, 3, 255), (3, 2, 257), (2, 7, 384),
                                           (1, 33, 511), (2, 32, 512), (3, 6, 513), (1, 1025, 641), (2, 9, 1025),
                                           (1, 2, 4099)])
def test_cauchy_at_tile_edges(rows, n, length):
    from lrnnx_b200.structured_kernels import cauchy_mult_sym_bwd, cauchy_mult_sym_fwd      # any number of poles
    v, z, w, g = _case(rows, n, length)
    on = [t.cuda() for t in (v, z, w, g)]
    out = cauchy_mult_sym_fwd(*on[:3])
    dv, dw = cauchy_mult_sym_bwd(*on)
    V, Z, W, G = (t.to(torch.cdouble) for t in (v, z, w, g))
    k1, k2 = 1 / (Z - W[..., None]), 1 / (Z - W[..., None].conj())              # (rows, n, length)
    V, G = V[..., None], G[:, None]
    # A term is exact up to the roundings of its factors: 1 for each of dr, e1, e2 and 3 for the squared modulus,
    # which enter it once or twice, 2 for the reciprocal and 3 for the products: at most 16, twice that with a
    # squared reciprocal.  Adding up m terms in any order costs m roundings of the sum of the moduli.
    want = {"out": (V * k1 + V.conj() * k2).sum(1), "dv": (G * k1.conj() + G.conj() * k2).sum(2),
            "dw": (V.conj() * (G * k1.conj() ** 2 + G.conj() * k2 ** 2)).sum(2)}
    size = {"out": (V.abs() * (k1.abs() + k2.abs())).sum(1), "dv": (G.abs() * (k1.abs() + k2.abs())).sum(2),
            "dw": (V.abs() * G.abs() * (k1.abs() ** 2 + k2.abs() ** 2)).sum(2)}
    # per-thread chains (2 terms per pole; 2 per 256 positions of a chunk), then 5 + 8 sums over lanes and warps and
    # the chunks (at least 1024 positions each)
    chain = length // 128 + 16 + length // 1024
    steps = {"out": 16 + 4 * n, "dv": 16 + chain, "dw": 36 + chain}
    for name, got in (("out", out), ("dv", dv), ("dw", dw)):
        err = (got.cpu().to(torch.cdouble) - want[name]).abs()
        bad = err > 2 * steps[name] * EPS * size[name]
        assert not bool(bad.any()), f"{name}: {int(bad.sum())} values outside, worst {float((err / size[name]).max()):.2e}"


def test_error_of_the_sums():
    """S4's points and poles: a pole enters the running sum with two roundings per part, which gives 1.7e-7 of the output
    (with four roundings it is 2.4e-7); the gradients' sums over the positions 1.2e-7 and 1.6e-7."""
    from lrnnx_b200.structured_kernels import cauchy_mult_sym_bwd, cauchy_mult_sym_fwd
    gen = torch.Generator().manual_seed(0)
    r = lambda *s: torch.randn(*s, generator=gen)
    rows, n, length = 64, 32, 4096
    omega = torch.exp(-2j * torch.pi * torch.arange(length, dtype=torch.float64) / (2 * length))
    z = (2 * (1 - omega) / (1 + omega)).to(torch.complex64)
    w = torch.complex(-0.025 * torch.exp(0.3 * r(rows, n)), 0.05 * torch.pi * torch.arange(n).float().expand(rows, n).contiguous())
    v, g = torch.complex(r(rows, n), r(rows, n)), torch.complex(r(rows, length), r(rows, length))
    v, z, w, g = (t.cuda() for t in (v, z, w, g))
    got = [cauchy_mult_sym_fwd(v, z, w), *cauchy_mult_sym_bwd(v, z, w, g)]
    V, Z, W, G = (t.to(torch.cdouble) for t in (v, z, w, g))
    k1, k2 = 1 / (Z - W[..., None]), 1 / (Z - W[..., None].conj())
    V, G = V[..., None], G[:, None]
    want = [(V * k1 + V.conj() * k2).sum(1), (G * k1.conj() + G.conj() * k2).sum(2), (V.conj() * (G * k1.conj() ** 2 + G.conj() * k2 ** 2)).sum(2)]
    for name, a, b in zip(("out", "dv", "dw"), got, want):
        err = float((a.to(torch.cdouble) - b).norm() / b.norm())
        assert err <= 2.0e-7, f"{name}: {err:.2e}"
