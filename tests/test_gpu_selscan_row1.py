"""The one-state-per-channel scan (RG-LRU, S7) where its tilings can go wrong: lengths around a lane's 8 steps,
a warp's 256, the row lengths at which the number of warps changes and the 2048-step chunks; constant B and C
other than 1; transitions close to 1, where sqrt(1 - a^2) cancels."""
from __future__ import annotations

import pytest
import torch

from conftest import assert_close
from oracle import scan_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["rglru", "s7"])
@pytest.mark.parametrize("L", [1, 7, 255, 256, 257, 512, 513, 1024, 1025, 2049, 4100])
def test_one_state_rows(method, L):
    from lrnnx_b200.ops import selective_scan_fn
    g = torch.Generator().manual_seed(L)
    batch, dim = 2, 5
    t = dict(u=torch.randn(batch, dim, L, generator=g), delta=torch.rand(batch, dim, L, generator=g) + 0.01,
             A=0.9 + 0.0999 * torch.rand(dim, 1, generator=g), B=torch.randn(dim, 1, generator=g), C=torch.randn(dim, 1, generator=g))
    gout = torch.randn(batch, dim, L, generator=g)
    names = ["u", "delta", "A", "B", "C"] if method == "rglru" else ["u", "delta", "B", "C"]

    def run(fn, cast, **kw):
        leaves = {k: cast(v).requires_grad_(True) for k, v in t.items()}
        out, last = fn(**leaves, return_last_state=True, discretization=method, **kw)
        grads = torch.autograd.grad(out, [leaves[k] for k in names], cast(gout))
        return [out.detach().cpu(), last.detach().cpu()] + [x.cpu() for x in grads]

    want = run(O.selective_scan_oracle, lambda v: v.double(), compute_dtype=torch.float64)
    got = run(selective_scan_fn, lambda v: v.cuda())
    # a product of up to a few hundred factors near 1, each with a rounding of 6e-8: 1e-4 leaves room for all of them
    for name, a, b in zip(["out", "last"] + ["d" + n for n in names], got, want):
        assert_close(a, b.float(), rtol=1e-4, atol_scale=2e-5, name=name)


@pytest.mark.parametrize("delta", [0.5, 1.0, 8.0])
def test_rglru_strong_decay(delta):
    """Transitions A**delta down to 1e-30, every row on its own scale (a row has one A).  Bound: a is exact relative to
    itself up to the rounding of x = delta log A, |x| 2^-24 <= 4e-6, and a few roundings of 6e-8; twice that.  u and
    dout are positive, so the sums that make dA do not cancel."""
    from lrnnx_b200.ops import rglru_scan_fn
    g = torch.Generator().manual_seed(7)
    A = torch.tensor([0.5, 0.3, 0.1, 0.05, 1e-2, 1e-3, 1e-4, 1e-6, 1e-7, 1e-8])
    A = A[A.double() ** (1.1 * delta) > 1e-30].unsqueeze(-1)
    shape = (2, A.shape[0], 300)
    u, dout = (0.75 + 0.5 * torch.rand(shape, generator=g) for _ in range(2))
    d = delta * (1 + 0.1 * torch.rand(shape, generator=g))

    def run(fn, cast, **kw):
        leaves = [cast(v).requires_grad_(True) for v in (u, d, A)]
        out = fn(*leaves, **kw)
        return [out.detach().cpu().double()] + [x.cpu().double() for x in torch.autograd.grad(out, leaves, cast(dout))]

    want = run(O.rglru_scan_oracle, lambda v: v.double(), compute_dtype=torch.float64)
    for name, a, b in zip(("out", "du", "ddelta", "dA"), run(rglru_scan_fn, lambda v: v.cuda()), want):
        err = (a - b).abs().amax(-1) / b.abs().amax(-1)
        assert float(err.max()) <= 1e-5, f"{name}: error by rows {err.tolist()}"
