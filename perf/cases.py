"""The work this framework is measured on: one pass per case through its public entry points.

Every case is what a user's program does with the library: a run of time steps
followed by the download of the state (`Context.step` + `download_fields`), the
same for a batch of small runs, the host-owned step, the statistics, the
allocation-free transform and the gradient of the learned closure.

`exact` restates each path in 64 bits with torch alone (torch.fft, no code of
this repository).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from hit3d_b200 import Context, Params
from hit3d_b200.batch import Batch
from hit3d_b200.gpu import Mlp, lib

TWO_PI = 2.0 * math.pi
PAIRS = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
FROB = (1.0, 2.0, 2.0, 1.0, 2.0, 1.0)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _dns(name, n, steps, **kw):
    """steps time steps in calls of `per_call` (0: one call), then the state's download.
    spectrum 2: k^2 exp(-2 (k/4)^2), the initial one of a DNS; 3: von Karman, a developed LES field.
    The FP32-transform form runs with launch variant 12 fixed, as a run's settings file fixes it where its
    results have to repeat to the last bit (the variants round differently in FP32); FP64 runs tune it."""
    c = dict(name=name, kind="dns", n=n, steps=steps, per_call=0, precision=0, dealias=0, forced=1, re=1000.0,
             dt=0.001, scalars=0, particles=0, les=0, spectrum=2)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: the allocation-free transform of one device field inside a host's time-critical loop
        dict(name="fft_static_48", kind="fft", n=48),
        # decaying DNS at 64^3, Re 400, one step per call as the host main loop makes them (Courant number read each step)
        _dns("decaying_64", 64, 20, per_call=1, forced=0, re=400.0, dt=0.005),
        # forced DNS at 256^3 with phase-shift dealiasing, two passive scalars and 10^6 cubic-interpolation particles
        _dns("phase_shift_256", 256, 20, dealias=1, scalars=2, particles=100),
        # the headline workload: forced DNS at 512^3, Re 3000, FP64
        _dns("forced_512", 512, 40, re=3000.0, dt=2e-4),
        # the same in the FP32-transform form
        _dns("forced_512_fp32", 512, 40, re=3000.0, dt=2e-4, precision=1),
        # 96 independent forced runs of four sizes, stepped together (training data of the closure)
        dict(name="batch_96", kind="batch", n32=32, n48=32, n64=28, n128=4, steps=50, graph=10),
        # LES at 128^3, Re 6000: Smagorinsky; the dynamic localization model (a transported k_sgs); the learned closure
        _dns("les_128_smagorinsky", 128, 50, les=1, re=6000.0, spectrum=3),
        _dns("les_128_dynamic", 128, 30, les=2, re=6000.0, spectrum=3),
        _dns("les_128_learned", 128, 50, les=20, re=6000.0, spectrum=3),
        # the statistics a run takes every IPRINT1 steps: velocity and two scalars at 256^3
        dict(name="stats_256", kind="stats", n=256, scalars=2, re=1000.0),
        # a host that owns its fields: 2/3-rule band up, one step, band down, eight states in flight
        dict(name="host_step_256", kind="host", n=256, inputs=8, re=1000.0, dt=0.001),
        # loss and gradient of the learned closure on one minibatch of its training
        dict(name="closure_gradient", kind="grad", points=16384, data=131072, lam=0.1),
    ]


def draw(rng):
    kind = rng.choice(["dns", "dns", "dns", "dns", "les", "les", "batch", "stats", "fft", "host", "grad"])
    re = round(10.0 ** rng.uniform(2.5, 3.8), 1)
    if kind == "fft":
        return dict(kind="fft", n=rng.choice([32, 48, 64, 128]))
    if kind == "grad":
        p = int(round(2.0 ** rng.uniform(8, 15)))
        return dict(kind="grad", points=p, data=4 * p + rng.randrange(1000), lam=rng.choice([0.0, 0.1]))
    if kind == "stats":
        return dict(kind="stats", n=rng.choice([48, 64, 128, 256]), scalars=rng.randrange(3), re=re)
    if kind == "host":
        n = rng.choice([48, 64, 128, 256])
        return dict(kind="host", n=n, inputs=rng.randrange(3, 10), re=re, dt=0.1 / n)
    if kind == "batch":
        return dict(kind="batch", n32=rng.randrange(1, 40), n48=rng.randrange(0, 40), n64=rng.randrange(0, 30),
                    n128=rng.randrange(0, 5), steps=rng.randrange(12, 50), graph=rng.choice([5, 10]))
    if kind == "les":
        n = rng.choice([32, 48, 64, 128])
        les = rng.choice([1, 1, 2, 20, 20])
        c = _dns("", n, rng.randrange(5, 40), les=les, re=re, dt=0.128 / n, spectrum=3,
                 precision=rng.randrange(2) if les == 1 else 0)
    else:
        n = rng.choice([32, 48, 64, 128, 256])
        precision = rng.choice([0, 0, 1])
        c = _dns("", n, rng.randrange(2, 30), forced=rng.choice([0, 1, 1]), re=re, dt=0.1 / n,
                 dealias=rng.choice([0, 0, 1]), precision=precision, scalars=rng.choice([0, 0, 1, 2]),
                 particles=0 if precision else rng.choice([0, 0, n // 4 + rng.randrange(9)]),
                 per_call=rng.choice([0, 0, 1]))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + salt) % (1 << 62))


def _axes(n):
    """Signed wavenumbers (N/2 stays positive), as (1,1,kx), (1,ky,1), (kz,1,1)."""
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    k = torch.where(2 * k > n, k - n, k)
    return k[: n // 2 + 1].view(1, 1, -1), k.view(1, -1, 1), k.view(-1, 1, 1)


def _initial(n, nf, seed, kmax, spectrum):
    """(nf, kz, ky, kx) complex: three solenoidal velocity components of energy 1 with the given
    spectrum, then scalars of the same spectrum with variance about 1 and mean 1/2; no mode beyond kmax."""
    g = _gen(seed)
    kx, ky, kz = _axes(n)
    k2 = kx * kx + ky * ky + kz * kz
    k = torch.sqrt(k2).clamp_(min=1.0)
    if spectrum == 2:
        amp = torch.exp(-((k / 4.0) ** 2))                              # sqrt(E / k^2)
    else:
        f2 = (TWO_PI * k / 4.0) ** 2
        amp = f2 / (1.0 + f2) ** 1.5 / k
    keep = (kx.abs() <= kmax) & (ky.abs() <= kmax) & (kz.abs() <= kmax) & (k2 > 0)
    amp = torch.where(keep, amp, torch.zeros_like(amp))
    u = torch.empty((nf, n, n, n // 2 + 1), dtype=torch.complex128, device="cuda")
    for f in range(nf):
        u[f] = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device="cuda", dtype=torch.float64))
        u[f] *= amp
    div = (kx * u[0] + ky * u[1] + kz * u[2]) / torch.where(k2 > 0, k2, torch.ones_like(k2))
    for f, kf in enumerate((kx, ky, kz)):
        u[f] -= kf * div
    w = torch.full((n // 2 + 1,), 1.0, device="cuda", dtype=torch.float64)
    w[0] = 0.5
    n3 = float(n) ** 3
    e = sum(float((w * (u[f].real ** 2 + u[f].imag ** 2)).sum()) for f in range(3)) / n3 ** 2
    u[:3] /= math.sqrt(e)
    for f in range(3, nf):
        e = float((w * (u[f].real ** 2 + u[f].imag ** 2)).sum()) / n3 ** 2
        u[f] /= math.sqrt(2.0 * e)
        u[f, 0, 0, 0] = 0.5 * n3
    return u


def _to_ref(u):
    """(nf, kz, ky, kx) complex -> the reference layout (nf, ky, kz, nx+2) float64, on the GPU."""
    r = torch.view_as_real(u.transpose(1, 2).contiguous())
    return r.reshape(r.shape[0], r.shape[1], r.shape[2], -1)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _host_fields(u):
    """The reference-layout host array (pinned, as a program that moves fields often keeps it)."""
    r = _to_ref(u)
    h = _pinned(r.shape)
    h.copy_(r)
    torch.cuda.synchronize()
    return h


def _kmax(case):
    n = case["n"]
    return int(math.floor(n / 3.0 * math.sqrt(2.0))) if case.get("dealias") and not case.get("les") else n // 3


def _particles(case, seed):
    """A particles^3 lattice displaced by a normal variate of n/16 cells (a cloud some time after its
    start on the lattice), in 1-based grid units."""
    n, m = case["n"], case["particles"]
    x = (torch.arange(m, device="cuda", dtype=torch.float64) + 0.5) * n / m
    z, y, x = torch.meshgrid(x, x, x, indexing="ij")
    p = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], dim=1)
    p = p + torch.randn(p.shape, generator=_gen(seed, 7), device="cuda", dtype=torch.float64) * (n / 16.0)
    return torch.remainder(p, float(n)) + 1.0


def _weights(n, delta, seed):
    """Closure parameters: Glorot-like layers, a small output layer, and an output bias near Smagorinsky's."""
    g = _gen(seed, 13)
    dx = TWO_PI / n
    out = []
    for nout, nin, scale in ((64, 6, 1.0), (64, 64, 1.0), (64, 64, 1.0), (5, 64, 0.01)):
        a = scale * math.sqrt(6.0 / (nin + nout))
        out.append((torch.rand(nout * nin, generator=g, device="cuda") * 2 - 1) * a)
        b = (torch.rand(nout, generator=g, device="cuda") * 2 - 1) * 0.05 * (nout == 64)
        if nout == 5:
            b[0] = -2.0 * 0.18 ** 2 * dx * dx / (delta * delta)
        out.append(b)
    return torch.cat(out)


def _closure_delta(n):
    return 2.0 * TWO_PI / n


def _closure_data(case, seed):
    """Traceless velocity gradients (9, P) and correlated stresses (6, P), float32, and the minibatch's indices."""
    g, p = _gen(seed, 17), case["data"]
    a = torch.randn((3, 3, p), generator=g, device="cuda")
    tr = (a[0, 0] + a[1, 1] + a[2, 2]) / 3.0
    for i in range(3):
        a[i, i] -= tr
    s = 0.5 * (a + a.transpose(0, 1))
    mag = torch.sqrt(2.0 * (s * s).sum((0, 1)))
    tau = torch.stack([-0.02 * mag * s[i, j] for i, j in PAIRS]) + 0.01 * torch.randn((6, p), generator=g, device="cuda")
    idx = torch.randint(0, p, (case["points"],), generator=g, device="cuda", dtype=torch.int32)
    return a.reshape(9, p), tau, idx


def _batch_runs(case):
    """[(n, Re, dt)] of the batch: Re over [200, 800], dt with the grid as the training runs have it."""
    runs = []
    for n in (32, 48, 64, 128):
        count = case["n%d" % n]
        runs += [(n, 200.0 + 600.0 * ((r * 0.618034) % 1.0), 0.004 * 64.0 / n) for r in range(count)]
    return runs


def _params(case, **kw):
    p = dict(nx=case["n"], dealias=0, flow_type=1, force_type=1, kfmax=2, famp=0.5, nu=1.0 / case.get("re", 1000.0),
             dt=case.get("dt", 0.001))
    p.update(kw)
    return Params(**p)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fft":
        n = case["n"]
        x = torch.zeros((n, n, n + 2), dtype=torch.float64, device="cuda")
        x[:, :, :n] = torch.randn((n, n, n), generator=_gen(seed), device="cuda", dtype=torch.float64)
        return dict(kind=kind, n=n, x=x, out=torch.empty_like(x), call=lib().hit3d_gpu_xfft3d_static)
    if kind == "grad":
        a, tau, idx = _closure_data(case, seed)
        m = Mlp()
        m.params = _weights(32, 1.0, seed).cpu().numpy()
        m.set_data(a.cpu().numpy(), tau.cpu().numpy(), 1.0)
        return dict(kind=kind, m=m, idx=idx.cpu().numpy(), lam=case["lam"])
    if kind == "batch":
        runs = _batch_runs(case)
        b = Batch([_params(dict(n=n, re=re, dt=dt)) for n, re, dt in runs])
        out = {}
        for n in (32, 48, 64, 128):
            mine = [r for r, q in enumerate(runs) if q[0] == n]
            if mine:
                h = _pinned((len(mine), 3, n, n, n + 2))
                for i, r in enumerate(mine):
                    h[i].copy_(_to_ref(_initial(n, 3, seed * 131 + r, n // 3, 2)))
                    torch.cuda.synchronize()
                    b.contexts[r].upload_fields(h[i].numpy())
                    b.contexts[r].dealias_all()
                out["n%d" % n] = (h, mine)
        b.autotune()
        return dict(kind=kind, b=b, out=out, steps=case["steps"], graph=case["graph"])
    if kind == "stats":
        ctx = Context(_params(case, n_scalars=case["scalars"], sc=[0.7, 1.0][: case["scalars"]],
                              scalar_type=[0] * case["scalars"]))
        ctx.upload_fields(_host_fields(_initial(case["n"], 3 + case["scalars"], seed, case["n"] // 3, 3)).numpy())
        return dict(kind=kind, ctx=ctx, scalars=case["scalars"])
    if kind == "host":
        ctx = Context(_params(case))
        ins = [_host_fields(_initial(case["n"], 3, seed * 31 + i, case["n"] // 3, 2)) for i in range(2)]
        outs = [torch.zeros_like(h, pin_memory=True) for h in ins]
        ctx.upload_fields(ins[0].numpy())
        ctx.autotune()
        return dict(kind=kind, ctx=ctx, outs=outs, ins=ins, i=[ins[q % 2].numpy() for q in range(case["inputs"])],
                    o=[outs[q % 2].numpy() for q in range(case["inputs"])])
    ns, les = case["scalars"], case["les"]
    ctx = Context(_params(case, dealias=case["dealias"], flow_type=case["forced"], precision=case["precision"],
                          les_model=les, n_scalars=ns, sc=[0.7, 1.0][:ns], scalar_type=[0] * ns))
    ctx.upload_fields(_host_fields(_initial(case["n"], 3 + ns, seed, _kmax(case), case["spectrum"])).numpy())
    if les == 20:
        d = _closure_delta(case["n"])
        bits = _weights(case["n"], d, seed).to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)
        ctx.les_set_mlp(bits, d, clip=True, kernel=1)
    if case["particles"]:
        ctx.particles_upload(_particles(case, seed).cpu().numpy(), None, scheme=1)
    ctx.dealias_all()
    if case["precision"] == 0:
        ctx.autotune()
    else:
        ctx.set_variant(12)
        ctx.set_column_tile(ctx.autotune_columns()[0])
    return dict(kind=kind, ctx=ctx, out=_pinned(ctx.field_shape()), steps=case["steps"], per_call=case["per_call"],
                particles=case["particles"])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "fft":
        x, out = state["x"], state["out"]
        rc = state["call"](state["n"], x.data_ptr(), out.data_ptr(),
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError("hit3d_gpu_xfft3d_static: code %d" % rc)
        return out
    if kind == "grad":
        loss, grad = state["m"].loss_grad(state["idx"], state["lam"])
        return {"loss": loss, "grad": grad}
    if kind == "batch":
        state["b"].step(state["steps"], graph_steps=state["graph"])
        for h, mine in state["out"].values():
            for i, r in enumerate(mine):
                state["b"].contexts[r].download_fields(out=h[i].numpy())
        return {k: h for k, (h, _) in state["out"].items()}
    if kind == "stats":
        ctx = state["ctx"]
        es, st = ctx.stats()
        return {"spectrum": es, "velocity": st, "scalars": [ctx.scalar_stats(s) for s in range(state["scalars"])]}
    if kind == "host":
        state["ctx"].step_host(state["i"], state["o"], nsteps=1, band_only=True)
        return state["outs"]
    ctx = state["ctx"]
    courant = 0.0
    if state["per_call"]:
        for _ in range(state["steps"]):
            courant = ctx.step(1)
    else:
        courant = ctx.step(state["steps"])
    ctx.download_fields(out=state["out"].numpy())
    out = {"fields": state["out"], "courant": courant}
    if state["particles"]:
        out["xyz"], out["uvw"] = ctx.particles_download()
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _step_work(n, steps, nf, nprod, passes, kept_all):
    """State and AB2 history read and written once per step at the modes the dealiasing keeps; the 3-D
    real transforms of `nf` inputs and `nprod` products, `passes` times (5/2 N^3 log2 N^3 each)."""
    kc = n // 3
    modes = n * n * (n // 2 + 1) if kept_all else (kc + 1) * (2 * kc + 1) ** 2
    return steps * 4 * nf * modes * 16.0, steps * passes * (nf + nprod) * 2.5 * n ** 3 * 3 * math.log2(n)


def work(case):
    kind = case["kind"]
    if kind == "fft":
        n = case["n"]
        return {"bytes": 2.0 * 8 * n * n * (n + 2), "flops": 7.5 * n ** 3 * math.log2(n)}
    if kind == "grad":
        p, w = case["points"], 6 * 64 + 2 * 64 * 64 + 5 * 64
        return {"bytes": p * (15 + 1) * 4.0 + 2 * (w + 197) * 4.0, "flops": 6.0 * p * w}
    if kind == "batch":
        b = f = 0.0
        for n, _, _ in _batch_runs(case):
            x, y = _step_work(n, case["steps"], 3, 6, 1, False)
            b, f = b + x + 3 * 8 * n * n * (n + 2), f + y
        return {"bytes": b, "flops": f}
    n = case["n"]
    if kind == "stats":
        nf = 3 + case["scalars"]
        return {"bytes": nf * 16.0 * n * n * (n // 2 + 1), "flops": (6 + 4 * case["scalars"]) * 7.5 * n ** 3 * math.log2(n)}
    if kind == "host":
        kc = n // 3
        b, f = _step_work(n, case["inputs"], 3, 6, 1, False)
        return {"bytes": b + case["inputs"] * 2 * 3 * 16.0 * (kc + 1) * (2 * kc + 1) ** 2, "flops": f}
    les = case["les"]
    nf = 3 + case["scalars"] + (1 if les == 2 else 0)
    b, f = _step_work(n, case["steps"], nf, 6 + 3 * (nf - 3), 2 if case["dealias"] and not les else 1,
                      bool(case["dealias"]) or les == 2)
    extra = {0: 0, 1: 12, 2: 20, 20: 15}[les] * case["steps"]
    return {"bytes": b + nf * 8.0 * n * n * (n + 2) + case["particles"] ** 3 * 96.0 * case["steps"],
            "flops": f + extra * 7.5 * n ** 3 * math.log2(n) + (les == 20) * case["steps"] * 2.0 * 8896 * n ** 3}


# ---------------------------------------------------------------------------
# the same in 64 bits with torch alone
# ---------------------------------------------------------------------------
def _features(a, delta):
    """Inputs x (6, P), basis t (5, 6, P), strain (6, P) and prefactor of the closure from a (3, 3, P)."""
    s, r = 0.5 * (a + a.transpose(0, 1)), 0.5 * (a - a.transpose(0, 1))
    strain = torch.stack([s[i, j] for i, j in PAIRS])
    mag = torch.sqrt(2.0 * (s * s).sum((0, 1))) + 1e-30
    s, r = s / mag, r / mag
    mm = lambda p, q: torch.einsum("ikp,kjp->ijp", p, q)  # noqa: E731
    tr = lambda p: p[0, 0] + p[1, 1] + p[2, 2]  # noqa: E731
    s2, r2 = mm(s, s), mm(r, r)
    x = torch.stack([tr(s2), tr(r2), tr(mm(s2, s)), tr(mm(s, r2)), tr(mm(s2, r2)),
                     torch.full_like(mag, delta * 32.0 / TWO_PI)])
    eye = torch.eye(3, device=a.device, dtype=a.dtype)[:, :, None]
    basis = [s, mm(s, r) - mm(r, s), s2 - eye * tr(s2) / 3.0, r2 - eye * tr(r2) / 3.0, mm(r, s2) - mm(s2, r)]
    t = torch.stack([torch.stack([b[i, j] for i, j in PAIRS]) for b in basis])
    return x, t, strain, delta * delta * mag * mag


def _network(w, x):
    o = 0
    for nout, nin in ((64, 6), (64, 64), (64, 64), (5, 64)):
        z = w[o:o + nout * nin].view(nout, nin) @ x + w[o + nout * nin:o + nout * nin + nout, None]
        o += nout * nin + nout
        x = z if nout == 5 else 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
    return x


def _closure_stress(w, a, delta):
    """Predicted stresses (6, P), zero where their dissipation is negative."""
    out = []
    for q in range(0, a.shape[2], 1 << 18):
        x, t, strain, pref = _features(a[:, :, q:q + (1 << 18)], delta)
        tau = pref * torch.einsum("np,ncp->cp", _network(w, x), t)
        diss = -sum(f * tau[c] * strain[c] for c, f in enumerate(FROB))
        out.append(torch.where(diss < 0, torch.zeros_like(tau), tau))
    return torch.cat(out, dim=1)


class _Flow:
    """The reference's time step (Euler, then Adams-Bashforth 2) in 64 bits."""

    def __init__(self, u, nu, dt, forced, dealias=0, pe=(), les=0, weights=None, xyz=None):
        self.u, self.nu, self.dt, self.forced, self.dealias, self.pe, self.les = u, nu, dt, forced, dealias, pe, les
        self.w, self.xyz, self.uvw, self.old, self.courant = weights, xyz, None, None, 0.0
        n = self.n = u.shape[1]
        self.dx = TWO_PI / n
        self.k = _axes(n)
        kx, ky, kz = self.k
        self.k2 = kx * kx + ky * ky + kz * kz
        self.alias = sum((q.abs() > n // 3).to(torch.int8) for q in self.k)
        sh = torch.round(torch.sqrt(self.k2.float()))
        self.band = (sh >= 1) & (sh <= 2) & (kx < n // 2)

    def phys(self, f):
        return torch.fft.irfftn(f, s=(self.n,) * 3, dim=(-3, -2, -1))

    def nonlinear(self, u):
        """-i k_j (u_i u_j)^ of the velocity and -i k_j (phi u_j)^ of every further field."""
        p = [self.phys(u[f]) for f in range(3)]
        r = [0, 0, 0]
        for i, j in PAIRS:
            q = torch.fft.rfftn(p[i] * p[j])
            r[i] = r[i] - 1j * self.k[j] * q
            if i != j:
                r[j] = r[j] - 1j * self.k[i] * q
        for f in range(3, u.shape[0]):
            phi = self.phys(u[f])
            r.append(sum(-1j * self.k[j] * torch.fft.rfftn(phi * p[j]) for j in range(3)))
        return r, p

    def strain(self):
        return [self.phys(0.5j * (self.k[j] * self.u[i] + self.k[i] * self.u[j])) for i, j in PAIRS]

    def stress(self, r, tau, keep):
        for c, (i, j) in enumerate(PAIRS):
            q = torch.fft.rfftn(tau[c]) * keep
            r[i] = r[i] - 1j * self.k[j] * q
            if i != j:
                r[j] = r[j] - 1j * self.k[i] * q

    def step(self):
        u, n = self.u, self.n
        nut = None
        if self.les == 2:
            ks = self.phys(torch.where(self.k2 > float(n // 3) ** 2, torch.zeros_like(u[3]), u[3]))
            low = float(ks.min())
            ks = ks.clamp(min=0.0)
            nut = 0.1 * self.dx * torch.sqrt(ks)
            if low < 0.0:
                u[3] = torch.fft.rfftn(ks)
        r, p = self.nonlinear(u)
        self.courant = float((p[0].abs() + p[1].abs() + p[2].abs()).max()) * self.dt / self.dx
        if self.xyz is not None:
            self.move(p)
        del p
        keep = self.alias == 0
        if self.dealias:
            keep = self.alias < 2
            ph = torch.exp(0.5j * self.dx * (self.k[0] + self.k[1] + self.k[2]))
            q, _ = self.nonlinear(u * ph)
            r = [0.5 * (a + b * ph.conj()) for a, b in zip(r, q)]
            del q, ph
        diff = [self.nu] * 3 + list(self.pe)
        for f in range(u.shape[0]):
            r[f] = torch.where(keep, r[f] - diff[f] * self.k2 * u[f], torch.zeros_like(r[f]))
        if self.les == 1:
            s = self.strain()
            nut = (0.18 * self.dx) ** 2 * torch.sqrt(2.0 * sum(f * s[c] ** 2 for c, f in enumerate(FROB)))
            self.stress(r, [-2.0 * nut * q for q in s], keep)
        elif self.les == 2:
            s = self.strain()
            self.stress(r, [-2.0 * nut * q for q in s], keep)
            cube = self.phys(torch.where(keep, u[3], torch.zeros_like(u[3]))).clamp(min=0.0)
            src = 2.0 * nut * sum(f * s[c] ** 2 for c, f in enumerate(FROB)) - cube ** 1.5 / self.dx
            r[3] = r[3] + torch.fft.rfftn(src) * keep
            for j in range(3):
                r[3] = r[3] + 1j * self.k[j] * torch.fft.rfftn(nut * self.phys(1j * self.k[j] * u[3])) * keep
        elif self.les == 20:
            a = torch.stack([torch.stack([self.phys(1j * self.k[j] * u[i]).reshape(-1) for j in range(3)]) for i in range(3)])
            tau = _closure_stress(self.w, a, _closure_delta(n))
            self.stress(r, [t.view(n, n, n) for t in tau], keep)
        if self.les == 0:
            for f in range(3, u.shape[0]):
                r[f] = r[f] - u[0]  # unit mean gradient along x
        if self.forced:
            half = torch.ones(n // 2 + 1, device="cuda", dtype=torch.float64)
            half[0] = 0.5
            e = sum(float(torch.where(self.band, half * (u[f].real ** 2 + u[f].imag ** 2), 0.0).sum()) for f in range(3))
            e /= float(n) ** 6
            for f in range(3):
                r[f] = r[f] + torch.where(self.band, 0.5 / e * u[f], torch.zeros_like(u[f]))
        for f in range(u.shape[0]):
            u[f] += self.dt * (r[f] if self.old is None else 1.5 * r[f] - 0.5 * self.old[f])
        self.old = r
        div = sum(self.k[f] * u[f] for f in range(3)) / torch.where(self.k2 > 0, self.k2, torch.ones_like(self.k2))
        for f in range(3):
            u[f] -= self.k[f] * div

    def move(self, p):
        """Four-point cubic (Lagrange) interpolation and Adams-Bashforth 2 in grid units."""
        n = self.n
        cell = torch.floor(self.xyz)
        t = self.xyz - cell
        i = cell.long() - 1
        wt = [-t * (t - 1) * (t - 2) / 6, (t + 1) * (t - 1) * (t - 2) / 2, -(t + 1) * t * (t - 2) / 2, (t + 1) * t * (t - 1) / 6]
        v = torch.zeros_like(self.xyz)
        for a in range(4):
            for b in range(4):
                for c in range(4):
                    at = (((i[:, 2] + a - 1) % n) * n + (i[:, 1] + b - 1) % n) * n + (i[:, 0] + c - 1) % n
                    f = wt[a][:, 2] * wt[b][:, 1] * wt[c][:, 0]
                    for d in range(3):
                        v[:, d] += f * p[d].reshape(-1)[at]
        rate = v if self.uvw is None else 1.5 * v - 0.5 * self.uvw
        self.uvw = v
        self.xyz = torch.remainder(self.xyz + rate * self.dt / self.dx - 1.0, float(n)) + 1.0


def _exact_stats(case, seed):
    n, nu = case["n"], 1.0 / case["re"]
    u = _initial(n, 3 + case["scalars"], seed, n // 3, 3)
    f = _Flow(u, nu, 0.0, 0)
    kx, ky, kz = f.k
    n6, kmax = float(n) ** 6, n // 3
    sh = torch.round(torch.sqrt(f.k2.float())).long().reshape(-1)
    half = torch.ones(n // 2 + 1, device="cuda", dtype=torch.float64)
    half[0] = 0.5
    half[-1] = 0.0

    def spectrum(fields):
        e = sum((half * (q.real ** 2 + q.imag ** 2)) for q in fields) / n6
        return torch.zeros(int(sh.max()) + 1, device="cuda", dtype=torch.float64).index_add_(0, sh, e.reshape(-1))[1:kmax + 1]

    es = spectrum(u[:3]).cpu().numpy()
    k = np.arange(1, kmax + 1)
    energy, eps = es.sum(), (es * k * k).sum() * 2.0 * nu
    eta, uvar = (nu ** 3 / eps) ** 0.25, 2.0 / 3.0 * energy
    xl, lam = math.pi / 2.0 * (es / k).sum() / uvar, math.sqrt(15.0 * uvar * nu / eps)
    w = [1j * (ky * u[2] - kz * u[1]), 1j * (kz * u[0] - kx * u[2]), 1j * (kx * u[1] - ky * u[0])]
    ens = float(sum((f.phys(q) ** 2).mean() for q in w))
    skew = 0.0
    for q in range(3):
        d = f.phys(1j * f.k[q] * u[q])
        skew += float((d ** 3).mean() / (d ** 2).mean() ** 1.5) / 3.0
    vel = {"energy": energy, "eps_v": eps, "eta": eta, "etakmax": eta * kmax, "uvar": uvar, "x_length": xl,
           "lambda": lam, "re_lambda": uvar * math.sqrt(15.0 / eps / nu), "re_lambda1": math.sqrt(uvar) * lam / nu,
           "tau_e": xl / math.sqrt(uvar), "enstrophy": ens, "skewness": skew}
    sc = []
    for s in range(case["scalars"]):
        phi = f.phys(u[3 + s])
        grad = float(sum((f.phys(1j * q * u[3 + s]) ** 2).mean() for q in f.k))
        sc.append(dict(spectrum=2.0 * spectrum(u[3 + s:4 + s]).cpu().numpy(), diss=2.0 * nu / [0.7, 1.0][s] * grad,
                       mean=float(phi.mean()), variance=float((phi ** 2).mean() - phi.mean() ** 2),
                       min=float(phi.min()), max=float(phi.max())))
    return {"spectrum": es, "velocity": {q: float(v) for q, v in vel.items()}, "scalars": sc}


def exact(case, seed):
    kind = case["kind"]
    if kind == "fft":
        n = case["n"]
        x = torch.randn((n, n, n), generator=_gen(seed), device="cuda", dtype=torch.float64)
        return _to_ref(torch.fft.rfftn(x)[None])[0]
    if kind == "grad":
        a, tau, idx = _closure_data(case, seed)
        w = _weights(32, 1.0, seed).to(torch.bfloat16).double().requires_grad_(True)
        a, tau = a.double().view(3, 3, -1), tau.double()
        tr = (tau[0] + tau[3] + tau[5]) / 3.0
        tau = torch.stack([t - tr if c in (0, 3, 5) else t for c, t in enumerate(tau)])
        frob = torch.tensor(FROB, device="cuda", dtype=torch.float64)[:, None]
        strain = torch.stack([0.5 * (a[i, j] + a[j, i]) for i, j in PAIRS])
        n1, n2 = 1.0 / (frob * tau * tau).sum(0).mean(), 1.0 / ((frob * tau * strain).sum(0) ** 2).mean()
        at = idx.long()
        x, t, strain, pref = _features(a[:, :, at], 1.0)
        e = pref * torch.einsum("np,ncp->cp", _network(w, x), t) - tau[:, at]
        loss = n1 * (frob * e * e).sum(0).mean() + case["lam"] * n2 * ((frob * e * strain).sum(0) ** 2).mean()
        loss.backward()
        return {"loss": float(loss), "grad": w.grad}
    if kind == "batch":
        runs, out = _batch_runs(case), {}
        for r, (n, re, dt) in enumerate(runs):
            f = _Flow(_initial(n, 3, seed * 131 + r, n // 3, 2), 1.0 / re, dt, 1)
            for _ in range(case["steps"]):
                f.step()
            out.setdefault("n%d" % n, []).append(_to_ref(f.u))
        return {k: torch.stack(v) for k, v in out.items()}
    if kind == "stats":
        return _exact_stats(case, seed)
    if kind == "host":
        ins = [_initial(case["n"], 3, seed * 31 + i, case["n"] // 3, 2) for i in range(2)]
        f, outs = _Flow(ins[0].clone(), 1.0 / case["re"], case["dt"], 1), [None, None]
        for q in range(case["inputs"]):
            f.u.copy_(ins[q % 2])
            f.step()
            outs[q % 2] = _to_ref(f.u)
        return outs
    n, les, nu = case["n"], case["les"], 1.0 / case["re"]
    u = _initial(n, 3 + case["scalars"], seed, _kmax(case), case["spectrum"])
    pe = [nu / s for s in (0.7, 1.0)[: case["scalars"]]]
    if les == 2:  # k_sgs = 0.1 at the start, diffused with the viscosity itself
        u = torch.cat([u, torch.zeros_like(u[:1])])
        u[3, 0, 0, 0] = 0.1 * float(n) ** 3
        pe = [nu]
    w = _weights(n, _closure_delta(n), seed).to(torch.bfloat16).double() if les == 20 else None
    f = _Flow(u, nu, case["dt"], case["forced"], 0 if les else case["dealias"], pe, les, w,
              _particles(case, seed) if case["particles"] else None)
    for _ in range(case["steps"]):
        f.step()
    out = {"fields": _to_ref(f.u), "courant": f.courant}
    if case["particles"]:
        out["xyz"], out["uvw"] = f.xyz, f.uvw
    return out
