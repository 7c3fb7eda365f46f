"""The performance cases of this package: what its users call, at the sizes they call it with.

Every case goes through a public entry point (``selective_scan_fn``, ``simplified_scan_fn``,
``rglru_scan_fn``, ``cauchy_mult``, ``selective_state_update``, ``MambaLMHeadModel``).  ``draw`` gives
further cases of the same kinds over the ranges below.

kind      what                                                     ranges
s6        selective scan, d_state 16, forward or forward+backward  batch 1..64, dim 64..5120 (multiples of 8), any length
ssu       one decoding step, d_state 16, state updated in place    batch 1..256, dim 256..5120, float32 / bfloat16 state
s5        projected diagonal complex scan, forward + backward      P 32..512, H 32..1024, any length, dirac / zoh / bilinear
rglru     RG-LRU scan, one state per channel, forward + backward   dim 128..2560, any length, float32
cauchy    S4 Cauchy kernel, forward + backward                     32 pole pairs, rows 64..1024, length 256..16384
lm        two-layer Mamba language model, loss and all gradients   length 64..1024
"""
import math

import torch
import torch.nn.functional as F

# --------------------------------------------------------------------------------------------- cases


def listed():
    return [
        # a small training call in float32 (a test-sized layer, a tiny model): launches and latency count
        dict(name="s6_small_f32", kind="s6", batch=2, dim=256, length=512, dtype="float32", z=True, grad=True, views=False),
        # one layer of the 130M Mamba language model in training, batch 8 x 2048 tokens
        dict(name="s6_layer_bf16", kind="s6", batch=8, dim=1536, length=2048, dtype="bfloat16", z=True, grad=True, views=False),
        # time series and audio batches are trained in float32 at whatever length the data has
        dict(name="s6_ragged_f32", kind="s6", batch=4, dim=776, length=1531, dtype="float32", z=False, grad=True, views=False),
        # the prefill of one layer of the 1.4B model: 64 prompts of 512 tokens, operands as views of the projections
        dict(name="s6_prefill_bf16", kind="s6", batch=64, dim=4096, length=512, dtype="bfloat16", z=True, grad=False, views=True),
        # one very long sequence through a layer of 2.8B width (forward only: scoring, embedding)
        dict(name="s6_long_bf16", kind="s6", batch=1, dim=5120, length=131072, dtype="bfloat16", z=True, grad=False, views=False),
        # the state update of one 1.4B layer per generated token, 64 sequences, bfloat16 cache
        dict(name="ssu_64_bf16", kind="ssu", batch=64, dim=4096, state="bfloat16", dtype="bfloat16"),
        # a single sequence decoding on the 130M model, float32 cache: the smallest call there is
        dict(name="ssu_1_f32", kind="ssu", batch=1, dim=1536, state="float32", dtype="bfloat16"),
        # S5 / LRU layer in training, batch 8 x 4096 steps, 256 states, 512 channels
        dict(name="s5_lti", kind="s5", batch=8, P=256, H=512, length=4096, disc="dirac"),
        # time-varying S5 on data of a length that is no multiple of anything
        dict(name="s5_ltv_ragged", kind="s5", batch=6, P=192, H=384, length=1999, disc="zoh"),
        # the recurrent layer of a Griffin-style model, 2 x 2048 tokens
        dict(name="rglru_layer", kind="rglru", batch=4, dim=1024, length=2048),
        # S4 layer: convolution kernels of 1024 rows at length 4096
        dict(name="cauchy_s4", kind="cauchy", rows=1024, poles=32, length=4096),
        # a whole training pass of a two-layer model of the 130M shape: logits, loss and every gradient
        dict(name="lm_2layer", kind="lm", batch=4, length=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["s6", "s6", "s6", "s6", "ssu", "s5", "rglru", "cauchy", "lm"])
    if kind == "s6":
        grad = rng.random() < 0.6
        while True:
            c = dict(kind=kind, batch=_log(rng, 1, 64), dim=8 * _log(rng, 8, 640), length=_log(rng, 32, 32768),
                     dtype=rng.choice(["float32", "bfloat16", "bfloat16", "float16"]), z=rng.random() < 0.75, grad=grad,
                     views=rng.random() < 0.3)
            if rng.random() < 0.5:
                c["length"] = max(32, c["length"] // 64 * 64)
            # the 64-bit recurrence walks the length step by step; the state of all steps is kept for the backward
            if c["batch"] * c["dim"] * c["length"] <= (1 << 25 if grad else 1 << 27):
                return c
    if kind == "ssu":
        return dict(kind=kind, batch=_log(rng, 1, 256), dim=8 * _log(rng, 32, 640), state=rng.choice(["float32", "bfloat16"]),
                    dtype=rng.choice(["float32", "bfloat16", "bfloat16"]))
    if kind == "s5":
        while True:
            c = dict(kind=kind, batch=_log(rng, 1, 16), P=8 * _log(rng, 4, 64), H=8 * _log(rng, 4, 128), length=_log(rng, 64, 16384),
                     disc=rng.choice(["dirac", "zoh", "bilinear"]))
            if rng.random() < 0.5:
                c["length"] = max(64, c["length"] // 64 * 64)
            if c["batch"] * max(c["P"], c["H"]) * c["length"] <= 1 << 24:
                return c
    if kind == "rglru":
        while True:
            c = dict(kind=kind, batch=_log(rng, 1, 16), dim=8 * _log(rng, 16, 320), length=_log(rng, 64, 16384))
            if rng.random() < 0.5:
                c["length"] = max(64, c["length"] // 64 * 64)
            if c["batch"] * c["dim"] * c["length"] <= 1 << 25:
                return c
    if kind == "cauchy":
        return dict(kind=kind, rows=_log(rng, 64, 1024), poles=32, length=_log(rng, 256, 16384))
    return dict(kind=kind, batch=rng.randint(1, 4), length=_log(rng, 64, 1024))


# -------------------------------------------------------------------------------------------- inputs


def _dt(name):
    return getattr(torch, name)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _inv_softplus_bias(g, dim):
    """The step-size bias of a Mamba layer: softplus(bias) log-uniform in [1e-3, 1e-1]."""
    dt = torch.exp(torch.rand(dim, generator=g, device="cuda") * (math.log(0.1) - math.log(1e-3)) + math.log(1e-3))
    return dt + torch.log(-torch.expm1(-dt))


def _randn(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def _prepare_s6(c, g):
    b, d, L, dt = c["batch"], c["dim"], c["length"], _dt(c["dtype"])
    N, R = 16, 48
    s = {"A": -torch.arange(1, N + 1, device="cuda", dtype=torch.float32).repeat(d, 1), "D": torch.ones(d, device="cuda"),
         "delta_bias": _inv_softplus_bias(g, d)}
    s["u"], s["delta"] = _randn(g, b, d, L, dtype=dt), _randn(g, b, d, L, dtype=dt)
    if c["views"]:       # as the layer calls it: z is a half of the input projection, B and C are rows of the second projection
        s["z"] = _randn(g, b, 2 * d, L, dtype=dt)[:, d:]
        x_dbl = _randn(g, b, R + 2 * N, L, dtype=dt)
        s["B"], s["C"] = x_dbl[:, R:R + N], x_dbl[:, R + N:]
    else:
        s["z"] = _randn(g, b, d, L, dtype=dt)
        s["B"], s["C"] = _randn(g, b, N, L, dtype=dt), _randn(g, b, N, L, dtype=dt)
    if not c["z"]:
        s["z"] = None
    if c["grad"]:
        s["dout"] = _randn(g, b, d, L, dtype=dt)
    return s


def _prepare_ssu(c, g):
    b, d, dt, N = c["batch"], c["dim"], _dt(c["dtype"]), 16
    return {"state": _randn(g, b, d, N).to(_dt(c["state"])), "x": _randn(g, b, d, dtype=dt), "dt": _randn(g, b, d, dtype=dt),
            "A": -torch.arange(1, N + 1, device="cuda", dtype=torch.float32).repeat(d, 1), "B": _randn(g, b, N, dtype=dt),
            "C": _randn(g, b, N, dtype=dt), "D": torch.ones(d, device="cuda"), "z": _randn(g, b, d, dtype=dt),
            "dt_bias": _inv_softplus_bias(g, d)}


def _prepare_s5(c, g):
    b, P, H, L = c["batch"], c["P"], c["H"], c["length"]
    lam = torch.polar(0.9 + 0.099 * torch.rand(P, generator=g, device="cuda"), math.pi / 10 * torch.rand(P, generator=g, device="cuda"))
    cn = lambda *shape: torch.complex(_randn(g, *shape), _randn(g, *shape)) / math.sqrt(2 * shape[-1])  # noqa: E731
    s = {"A": torch.log(lam), "B": cn(P, H), "C": cn(H, P), "u": torch.complex(_randn(g, b, H, L), torch.zeros(b, H, L, device="cuda"))}
    # the time-invariant layer steps by one; the time-varying ones by a step size that the data chooses
    s["delta"] = torch.ones(b, P, L, device="cuda") if c["disc"] == "dirac" else 0.5 + torch.rand(b, P, L, generator=g, device="cuda")
    s["dout"] = torch.complex(_randn(g, b, H, L), _randn(g, b, H, L))
    return s


def _prepare_rglru(c, g):
    b, d, L = c["batch"], c["dim"], c["length"]
    # a = sigmoid(Lambda) in [0.9, 0.999], delta = 8 * gate as in the recurrent block
    A = 0.9 + 0.099 * torch.rand(d, 1, generator=g, device="cuda")
    return {"u": _randn(g, b, d, L), "delta": 8 * torch.sigmoid(_randn(g, b, d, L)), "A": A, "dout": _randn(g, b, d, L)}


def _prepare_cauchy(c, g):
    n, L = c["poles"], c["length"]
    # S4: evaluation points of the bilinear transform at the roots of unity, poles in the left half plane
    omega = torch.exp(-2j * math.pi * torch.arange(L, device="cuda", dtype=torch.float64) / (2 * L))
    z = (2 * (1 - omega) / (1 + omega)).to(torch.complex64)
    w = torch.complex(-0.5 * torch.exp(0.3 * _randn(g, c["rows"], n)) * 0.05,
                      0.05 * math.pi * torch.arange(n, device="cuda", dtype=torch.float32).expand(c["rows"], n).contiguous())
    return {"v": torch.complex(_randn(g, c["rows"], n), _randn(g, c["rows"], n)), "z": z, "w": w,
            "dout": torch.complex(_randn(g, c["rows"], L), _randn(g, c["rows"], L))}


_LM = dict(d_model=768, n_layer=2, vocab_size=50280)


def _prepare_lm(c, g):
    from lrnnx_b200.lm import MambaLMHeadModel
    with torch.random.fork_rng(devices=[torch.cuda.current_device()]):
        torch.manual_seed(int(torch.randint(1 << 30, (1,), generator=g, device="cuda")))
        model = MambaLMHeadModel(**_LM, device="cuda", dtype=torch.bfloat16)
    ids = torch.randint(_LM["vocab_size"], (c["batch"], c["length"]), generator=g, device="cuda")
    return {"model": model, "ids": ids}


def prepare(case, seed):
    return {"case": case, **globals()["_prepare_" + case["kind"]](case, _gen(seed))}


# ----------------------------------------------------------------------------------------- the calls

_S6_ARGS = ("u", "delta", "A", "B", "C", "D", "z", "delta_bias")


def _run_s6(s):
    from lrnnx_b200.ops.selective_scan import selective_scan_fn
    c = s["case"]
    args = [s[k] for k in _S6_ARGS]
    if not c["grad"]:
        with torch.no_grad():
            return selective_scan_fn(*args, delta_softplus=True, return_last_state=c["views"])
    args = [None if t is None else t.detach().requires_grad_() for t in args]
    out = selective_scan_fn(*args, delta_softplus=True)
    return [out] + list(torch.autograd.grad(out, [t for t in args if t is not None], s["dout"]))


def _run_ssu(s):
    from lrnnx_b200.ops.selective_state_update import selective_state_update
    # the state decays towards its inputs, so any number of steps on the same token keeps it in range
    out = selective_state_update(s["state"], s["x"], s["dt"], s["A"], s["B"], s["C"], s["D"], s["z"], s["dt_bias"], True)
    return [out, s["state"]]


def _run_s5(s):
    from lrnnx_b200.ops.simplified_scan import simplified_scan_fn
    args = [s[k].detach().requires_grad_() for k in ("u", "delta", "A", "B", "C")]
    y = simplified_scan_fn(*args, discretization=s["case"]["disc"])
    return [y] + list(torch.autograd.grad(y, args, s["dout"]))


def _run_rglru(s):
    from lrnnx_b200.ops.rglru_scan import rglru_scan_fn
    args = [s[k].detach().requires_grad_() for k in ("u", "delta", "A")]
    y = rglru_scan_fn(*args)
    return [y] + list(torch.autograd.grad(y, args, s["dout"]))


def _run_cauchy(s):
    from lrnnx_b200.ops.s4 import cauchy_mult
    v, w = s["v"].detach().requires_grad_(), s["w"].detach().requires_grad_()
    y = cauchy_mult(v, s["z"], w)
    return [y] + list(torch.autograd.grad(y, [v, w], s["dout"]))


def _run_lm(s):
    from lrnnx_b200.ops.cross_entropy import cross_entropy
    model, ids = s["model"], s["ids"]
    logits = model(ids)
    loss = cross_entropy(logits.view(-1, logits.shape[-1]), F.pad(ids[:, 1:], (0, 1), value=-100).view(-1))
    names, params = zip(*[(n, p) for n, p in model.named_parameters()])
    return {"logits": logits, "loss": loss, "grads": dict(zip(names, torch.autograd.grad(loss, params)))}


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


# ------------------------------------------------------------------------- what a pass has to move


def work(case):
    c, k = case, case["kind"]
    if k == "s6":
        n, s, N = c["batch"] * c["dim"] * c["length"], _dt(c["dtype"]).itemsize, 16
        bc = 2 * c["batch"] * N * c["length"]
        acts = 3 + c["z"]                       # u, delta, (z) in, out written
        fwd_b, fwd_f = s * (acts * n + bc), n * N * 6
        if not c["grad"]:
            return {"bytes": fwd_b + 8 * c["dim"] * N, "flops": fwd_f}
        # backward: the same operands and dout read again, their gradients written
        return {"bytes": fwd_b + s * (2 * (2 + c["z"]) * n + n + 2 * bc), "flops": fwd_f + n * N * 16}
    if k == "ssu":
        n = c["batch"] * c["dim"]
        return {"bytes": 2 * 16 * n * _dt(c["state"]).itemsize + 4 * n * _dt(c["dtype"]).itemsize + 4 * 18 * c["dim"], "flops": 6 * 16 * n}
    if k == "s5":
        nu, nx = c["batch"] * c["H"] * c["length"], c["batch"] * c["P"] * c["length"]
        # u, delta, dout in; y, du, ddelta out; the two projections, their transposes and the two weight gradients
        return {"bytes": 8 * 4 * nu + 4 * 2 * nx + 4 * 8 * c["P"] * c["H"], "flops": 6 * 8 * nx * c["H"] + 60 * nx}
    if k == "rglru":
        n = c["batch"] * c["dim"] * c["length"]
        return {"bytes": 4 * 3 * n + 4 * 5 * n, "flops": 30 * n}
    if k == "cauchy":
        return {"bytes": 8 * 2 * c["rows"] * c["length"] + 8 * 4 * c["rows"] * c["poles"], "flops": 96 * c["rows"] * c["length"] * c["poles"]}
    d, v, n = _LM["d_model"], _LM["vocab_size"], c["batch"] * c["length"]
    per_layer = 3 * d * 2 * d + 2 * d * (48 + 32) + 48 * 2 * d
    weights = v * d + _LM["n_layer"] * per_layer
    # weights read twice and their gradients written, logits written and their gradient read
    return {"bytes": 2 * 3 * weights + 2 * 2 * n * v, "flops": 6 * n * weights + _LM["n_layer"] * n * 2 * d * 16 * 22}


def tolerance(case):
    """About four times the error against 64 bits that was measured: 16-bit outputs are rounded to 8 or 11 bits; the
    S5 rows remember about a thousand steps, over which rounding in the products of coefficients adds up."""
    k = case["kind"]
    if k == "lm":
        return {"rel": 3e-2}
    if "bfloat16" in (case.get("dtype"), case.get("state")):
        return {"rel": 1e-2}
    if case.get("dtype") == "float16":
        return {"rel": 2e-3}
    return {"rel": {"s6": 2e-5, "ssu": 2e-6, "s5": 2e-4, "rglru": 2e-5, "cauchy": 2e-6}[k]}


# ------------------------------------------------------------------------------- the same in 64 bits


def _scan64(a_of, b_of, L, shape, dtype, keep):
    """h_t = a_t h_{t-1} + b_t over t in blocks of 64 coefficients; every state if ``keep``, else a callback sees each block."""
    h = torch.zeros(shape, device="cuda", dtype=dtype)
    out = []
    for t0 in range(0, L, 64):
        t1 = min(L, t0 + 64)
        a, b = a_of(t0, t1), b_of(t0, t1)
        blk = []
        for i in range(t1 - t0):
            h = torch.addcmul(b[i], a[i], h)
            blk.append(h)
        out.append(keep(t0, t1, torch.stack(blk)))
    return out, h


def _exact_s6(c, s):
    if c["batch"] * c["dim"] * c["length"] * (6 if c["grad"] else 1) > 1 << 30 or c["length"] > 140000:
        return None
    f = lambda t: None if t is None else t.double()  # noqa: E731
    b, d, L = c["batch"], c["dim"], c["length"]
    A, D, bias = f(s["A"]), f(s["D"]), f(s["delta_bias"])
    tm = lambda t, t0, t1: t[..., t0:t1].permute(2, 0, 1).double()  # noqa: E731   (steps, batch, rows)
    dts = lambda t0, t1: F.softplus(tm(s["delta"], t0, t1) + bias)  # noqa: E731
    a_of = lambda t0, t1: torch.exp(dts(t0, t1).unsqueeze(-1) * A)  # noqa: E731
    b_of = lambda t0, t1: (dts(t0, t1) * tm(s["u"], t0, t1)).unsqueeze(-1) * tm(s["B"], t0, t1).unsqueeze(2)  # noqa: E731
    dev, states = dict(device="cuda", dtype=torch.float64), []
    y = torch.empty(b, d, L, device="cuda", dtype=torch.float64 if c["grad"] else torch.float32)

    def keep(t0, t1, h):
        yy = torch.einsum("tbdn,tbn->bdt", h, tm(s["C"], t0, t1))
        yy += D[:, None] * s["u"][..., t0:t1].double()
        if c["grad"]:
            states.append(h)
        elif s["z"] is not None:
            yy *= F.silu(s["z"][..., t0:t1].double())
        y[..., t0:t1] = yy

    _, last = _scan64(a_of, b_of, L, (b, d, 16), torch.float64, keep)
    if not c["grad"]:
        return (y, last) if c["views"] else y
    z, dout = f(s["z"]), f(s["dout"])
    dy, dz, out = dout, None, y
    if z is not None:
        sg = torch.sigmoid(z)
        dy, dz, out = dout * z * sg, dout * y * sg * (1 + z * (1 - sg)), y * z * sg
    du, dd = torch.empty(b, d, L, **dev), torch.empty(b, d, L, **dev)
    dB, dC = torch.empty(b, 16, L, **dev), torch.empty(b, 16, L, **dev)
    dA, q = torch.zeros(d, 16, **dev), torch.zeros(b, d, 16, **dev)
    for k in reversed(range(len(states))):
        t0 = 64 * k
        t1 = min(L, t0 + 64)
        h, a = states[k], a_of(t0, t1)
        first = states[k - 1][-1:] if k else torch.zeros_like(h[:1])
        hp = torch.cat([first, h[:-1]])
        dyb, Bb, Cb, dtb, ub = tm(dy, t0, t1), tm(s["B"], t0, t1), tm(s["C"], t0, t1), dts(t0, t1), tm(s["u"], t0, t1)
        seed = dyb.unsqueeze(-1) * Cb.unsqueeze(2)
        g = []
        for i in reversed(range(t1 - t0)):
            gi = seed[i] + q
            g.append(gi)
            q = a[i] * gi
        g = torch.stack(g[::-1])
        ga = g * a * hp
        dA += torch.einsum("tbdn,tbd->dn", ga, dtb)
        gB = torch.einsum("tbdn,tbn->tbd", g, Bb)
        dtg = torch.einsum("tbdn,dn->tbd", ga, A) + gB * ub
        dd[..., t0:t1] = (dtg * torch.sigmoid(tm(s["delta"], t0, t1) + bias)).permute(1, 2, 0)
        du[..., t0:t1] = (gB * dtb + D * dyb).permute(1, 2, 0)
        dB[..., t0:t1] = torch.einsum("tbdn,tbd->bnt", g, dtb * ub)
        dC[..., t0:t1] = torch.einsum("tbdn,tbd->bnt", h, dyb)
        states[k] = states[k][-1:]
    grads = [du, dd, dA, dB, dC, (dy * f(s["u"])).sum((0, 2))] + ([] if dz is None else [dz]) + [dd.sum((0, 2))]
    return [out] + grads


def _exact_ssu(c, s):
    f = {k: (v.double() if torch.is_tensor(v) else v) for k, v in s.items()}
    dt = F.softplus(f["dt"] + f["dt_bias"])
    st = f["state"] * torch.exp(dt.unsqueeze(-1) * f["A"]) + (dt * f["x"]).unsqueeze(-1) * f["B"].unsqueeze(1)
    y = (st * f["C"].unsqueeze(1)).sum(-1) + f["D"] * f["x"]
    return [y * F.silu(f["z"]), st]


def _gain64(disc, A, d):
    """The transition, the input gain, and both derivatives of each (with respect to A d and A, d)."""
    x = A * d
    if disc == "dirac":
        a = torch.exp(x)
        return a, torch.ones_like(a), d * a, A * a, torch.zeros_like(a), torch.zeros_like(a)
    if disc == "zoh":
        a = torch.exp(x)
        k = (a - 1) / A
        return a, k, d * a, A * a, (d * a - k) / A, a
    r = 1 / (1 - 0.5 * x)
    return (1 + 0.5 * x) * r, d * r, d * r * r, A * r * r, 0.5 * d * d * r * r, r + 0.5 * d * A * r * r


def _exact_s5(c, s):
    b, P, L = c["batch"], c["P"], c["length"]
    w = lambda t: t.to(torch.complex128)  # noqa: E731
    A, B, C, u, dout = (w(s[k]) for k in ("A", "B", "C", "u", "dout"))
    d = s["delta"].double().permute(2, 0, 1)
    bu = torch.einsum("ph,bhl->lbp", B, u)
    a_of = lambda t0, t1: _gain64(c["disc"], A, d[t0:t1])[0]  # noqa: E731
    b_of = lambda t0, t1: _gain64(c["disc"], A, d[t0:t1])[1] * bu[t0:t1]  # noqa: E731
    hs, _ = _scan64(a_of, b_of, L, (b, P), torch.complex128, lambda t0, t1, h: h)
    h = torch.cat(hs)
    y = torch.einsum("hp,lbp->bhl", C, h)
    dC = torch.einsum("bhl,lbp->hp", dout, h.conj())
    seed = torch.einsum("hp,bhl->lbp", C.conj(), dout)
    q, g = torch.zeros(b, P, device="cuda", dtype=torch.complex128), torch.empty_like(h)
    for t1 in range(L, 0, -64):
        t0 = max(0, t1 - 64)
        ac = a_of(t0, t1).conj()
        for i in reversed(range(t1 - t0)):
            g[t0 + i] = seed[t0 + i] + q
            q = ac[i] * g[t0 + i]
    hp = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    a, k, da_dA, da_dd, dk_dA, dk_dd = _gain64(c["disc"], A, d)
    ga, gk = g * hp.conj(), g * bu.conj()
    dA = (ga * da_dA.conj() + gk * dk_dA.conj()).sum((0, 1))
    dd = (ga * da_dd.conj() + gk * dk_dd.conj()).real.permute(1, 2, 0)
    dbu = g * k.conj()
    return [y, torch.einsum("ph,lbp->bhl", B.conj(), dbu), dd, dA, torch.einsum("lbp,bhl->ph", dbu, u.conj()), dC]


def _exact_rglru(c, s):
    A, u, d, dout = (s[k].double() for k in ("A", "u", "delta", "dout"))
    lA = torch.log(A[:, 0])
    d, u, dout = (t.permute(2, 0, 1) for t in (d, u, dout))
    a = torch.exp(d * lA)
    b = torch.sqrt(1 - a * a)
    hs, _ = _scan64(lambda t0, t1: a[t0:t1], lambda t0, t1: b[t0:t1] * u[t0:t1], c["length"], u.shape[1:], torch.float64, lambda t0, t1, h: h)
    h = torch.cat(hs)
    g, q = torch.empty_like(h), torch.zeros_like(h[0])
    for i in reversed(range(c["length"])):
        g[i] = dout[i] + q
        q = a[i] * g[i]
    hp = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    da = g * hp - g * u * a / b
    y, du, dd = (t.permute(1, 2, 0) for t in (h, g * b, da * a * lA))
    return [y, du, dd, (da * a * d).sum((0, 1)).unsqueeze(-1) / A]


def _exact_cauchy(c, s):
    v, z, w, dout = (s[k].to(torch.complex128) for k in ("v", "z", "w", "dout"))
    y, dv, dw = torch.empty_like(dout), torch.empty_like(v), torch.empty_like(w)
    for r in range(0, c["rows"], 32):
        vv, ww = v[r:r + 32].unsqueeze(1), w[r:r + 32].unsqueeze(1)
        r1, r2, do = 1 / (z[:, None] - ww), 1 / (z[:, None] - ww.conj()), dout[r:r + 32].unsqueeze(-1)
        y[r:r + 32] = (vv * r1 + vv.conj() * r2).sum(-1)
        dv[r:r + 32] = (do * r1.conj() + do.conj() * r2).sum(1)
        dw[r:r + 32] = (do * (vv * r1 * r1).conj() + do.conj() * (vv.conj() * r2 * r2)).sum(1)
    return [y, dv, dw]


class _Scan64(torch.autograd.Function):
    """y_t = C_t . h_t of h_t = a_t h_{t-1} + x_t with tensors (L, batch, rows, states): a plain loop, and its adjoint loop."""

    @staticmethod
    def forward(ctx, a, x):
        h, out = torch.zeros_like(a[0]), torch.empty_like(a)
        for t in range(a.shape[0]):
            h = torch.addcmul(x[t], a[t], h)
            out[t] = h
        ctx.save_for_backward(a, out)
        return out

    @staticmethod
    def backward(ctx, dh):
        a, out = ctx.saved_tensors
        g, q = torch.empty_like(a), torch.zeros_like(a[0])
        for t in reversed(range(a.shape[0])):
            g[t] = dh[t] + q
            q = a[t] * g[t]
        hp = torch.cat([torch.zeros_like(out[:1]), out[:-1]])
        return g * hp, g


def _exact_lm(c, s):
    p = {n: t.detach().double().requires_grad_() for n, t in s["model"].named_parameters()}
    ids, emb = s["ids"], p["backbone.embedding.weight"]
    norm = lambda x, w: x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w  # noqa: E731
    res = F.embedding(ids, emb)
    for i in range(_LM["n_layer"]):
        q = lambda n: p["backbone.layers.%d.mixer.%s" % (i, n)]  # noqa: B023,E731
        xz = norm(res, p["backbone.layers.%d.norm.weight" % i]) @ q("in_proj.weight").t()
        x, z = xz.chunk(2, dim=-1)
        w = q("conv1d.weight")
        x = F.silu(F.conv1d(x.transpose(1, 2), w, q("conv1d.bias"), padding=w.shape[-1] - 1, groups=w.shape[0])[..., :ids.shape[1]]).transpose(1, 2)
        r, n = q("dt_proj.weight").shape[1], q("A_log").shape[1]
        dt, B, C = (x @ q("x_proj.weight").t()).split([r, n, n], dim=-1)
        dt = F.softplus(dt @ q("dt_proj.weight").t() + q("dt_proj.bias")).transpose(0, 1)        # (L, batch, d)
        tl = lambda t: t.transpose(0, 1)  # noqa: E731
        h = _Scan64.apply(torch.exp(dt.unsqueeze(-1) * -torch.exp(q("A_log"))), (dt * tl(x)).unsqueeze(-1) * tl(B).unsqueeze(2))
        y = torch.einsum("tbdn,tbn->btd", h, tl(C)) + x * q("D")
        res = res + (y * F.silu(z)) @ q("out_proj.weight").t()
    logits = norm(res, p["backbone.norm_f.weight"]) @ emb.t()
    loss = F.cross_entropy(logits[:, :-1].reshape(-1, logits.shape[-1]), ids[:, 1:].reshape(-1))
    return {"logits": logits.detach(), "loss": loss.detach(), "grads": dict(zip(p, torch.autograd.grad(loss, list(p.values()))))}


def exact(case, seed):
    s = prepare(case, seed)
    if case["kind"] == "lm":
        return _exact_lm(case, s)
    with torch.no_grad():
        return globals()["_exact_" + case["kind"]](case, s)
