"""Performance cases of the gSQG framework: the calls a simulation program makes.

Every case is a dict of plain values; ``prepare`` builds what the program has in
hand on the GPU, ``run`` makes one pass through the public entry points and
``exact`` gives the same outputs from plain torch in float64.

Fields.  "fresh" states come from ``initialize`` on a physical field, as a run
begins (every mode carries at least round-off).  "running" states are spectra of
a run in progress, as a checkpoint or the previous call leaves them: the modes
outside the 2/3 dealiasing disk get no tendency, and hyperviscosity has removed
what they once held.
"""

import math
import os

import numpy as np
import torch

import pygsquig_b200 as P
from pygsquig_b200.closure.cnn import ClosureCNN
from pygsquig_b200.closure.model import ClosureSolver, SubgridClosure
from pygsquig_b200.ensemble import EnsembleSolver, Member

TWO_PI = 2 * math.pi
C128 = torch.complex128
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(P.__file__)), "closure", "trained", "closure_weights.npz")


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------


def _flow(name, kind, N, precision, **kw):
    """A call on one field.  Defaults: SQG, integrating-factor RK4, no forcing."""
    c = dict(name=name, kind=kind, N=N, precision=precision, L=TWO_PI, alpha=1.0, scheme="ifrk4", nu=0.0, p=8,
             mu=0.0, kf=0.0, dk=2.0, eps=0.1, dt=1e-3, steps=1, scalars=0, source=False, kappa=1e-4,
             spectrum="k4exp", start="fresh")
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: one explicit step of an inviscid test problem
        _flow("step_n64_f64", "step", 64, "float64", scheme="explicit", dt=2e-3),
        # decaying SQG at a laptop-sized grid, stepped one call at a time
        _flow("plain_n256_f64", "step", 256, "float64", nu=1e-4, spectrum="sines"),
        # a right-hand side for a program's own integrator (SSP-RK3 and the like)
        _flow("rhs_n512_f64", "rhs", 512, "float64", nu=1e-18, alpha=0.5, start="running"),
        # a physical field in, its velocity out: initialisation and output of a run
        _flow("transforms_n2048_f32", "transforms", 2048, "float32", alpha=1.3),
        # forced-dissipative runs between two outputs, both precisions
        _flow("forced_n1024_f32", "multistep", 1024, "float32", nu=1e-8, mu=0.1, kf=40.0, dt=2e-4, steps=10),
        _flow("forced_n1024_f64", "multistep", 1024, "float64", nu=1e-8, mu=0.1, kf=40.0, dt=2e-4, steps=5),
        # the DNS behind the learned closure, a few steps between two samples
        _flow("dns_n2048_f32", "multistep", 2048, "float32", nu=1e-22, mu=0.1, kf=20.0, dt=1e-4, steps=4,
              start="running"),
        # the largest run: ring forcing and two mean-gradient scalars, in both precisions
        _flow("hires_n4096_f32", "step", 4096, "float32", alpha=0.5, nu=1e-20, mu=0.05, kf=100.0, dt=5e-5, scalars=2,
              source=True, spectrum="kminus3", start="running"),
        _flow("hires_n4096_f64", "step", 4096, "float64", alpha=0.5, nu=1e-20, mu=0.05, kf=100.0, dt=5e-5, scalars=2,
              source=True, spectrum="kminus3", start="fresh"),
        # an ensemble of uneven sizes, alphas and scalar counts
        dict(name="ensemble96_f32", kind="ensemble", precision="float32", layout=7, n128=48, n256=32, n512=16,
             nu=1e-6, p=8, dt=5e-4, steps=5),
        # the coarse solve with the trained closure on every RK stage
        dict(name="closure_solve_n256", kind="closure_solve", N=256, precision="float32", steps=4, substeps=10,
             dt=1e-3, nu=1e-22, p=8, mu=0.1, kf=20.0, dk=2.0, eps=0.1, alpha=1.0, L=TWO_PI),
        # one optimiser step of the closure network
        dict(name="closure_train_b16", kind="closure_train", size=256, batch=16),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "multistep", "multistep", "rhs", "transforms", "ensemble", "closure_train"])
    if kind == "ensemble":
        sizes = sorted(rng.sample([32, 64, 128, 256, 512], rng.randint(1, 3)))
        return dict(kind=kind, precision=rng.choice(["float32", "float32", "float64"]), layout=rng.randint(0, 10**6),
                    **{f"n{n}": rng.randint(1, max(2, 48 * 128 // n)) for n in sizes},
                    nu=10 ** rng.uniform(-14, -6), p=8, dt=rng.uniform(1e-4, 5e-4), steps=rng.randint(2, 5))
    if kind == "closure_train":
        return dict(kind=kind, size=rng.choice([128, 256, 384]), batch=rng.randint(1, 7))
    N = 1 << rng.randint(3, 12)
    prec = rng.choice(["float32", "float64"])
    if N == 4096 and kind == "multistep":
        prec = "float32"
    alpha = rng.choice([0.0, 0.5, 1.0, 1.5, 2.0, round(rng.uniform(0.1, 1.9), 3)])
    p = rng.choice([2, 4, 8])
    L = rng.choice([TWO_PI, TWO_PI, 1.0, rng.uniform(2.0, 12.0)])
    k1 = TWO_PI / L
    kc = k1 * N / 3.0
    dt = rng.uniform(0.02, 0.1) * (L / N) / max(1.0, (6 * k1) ** (1 - alpha))
    scheme = rng.choice(["ifrk4", "ifrk4", "explicit"])
    # viscous rate at the dealiasing radius times dt: stable for the explicit scheme
    rate = 10 ** rng.uniform(-3, -0.7) if scheme == "explicit" else 10 ** rng.uniform(-3, 3)
    forced = N >= 64 and rng.random() < 0.6
    scalars = rng.randint(0, 2) if kind == "step" else 0
    return _flow("", kind, N, prec, L=L, alpha=alpha, p=p, dt=dt, scheme=scheme, nu=rate / dt / kc**p,
                 mu=rng.choice([0.0, 0.1]), kf=k1 * rng.uniform(3.0, N / 12.0) if forced else 0.0, dk=2.0 * k1,
                 steps=1 if kind != "multistep" else (2 if N == 4096 else rng.randint(2, 10)),
                 scalars=scalars, source=bool(scalars and rng.random() < 0.5), kappa=10 ** rng.uniform(-6, -3),
                 spectrum=rng.choice(["k4exp", "kminus3"]), start=rng.choice(["fresh", "running"]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _rdtype(case):
    return torch.float64 if case["precision"] == "float64" else torch.float32


def _k1d(N, L):
    return torch.as_tensor(np.fft.fftfreq(N, d=L / N) * 2 * np.pi, device="cuda")


def _k2(N, L):
    k = _k1d(N, L)
    return k[:, None] ** 2 + k[None, :] ** 2


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _random_field(N, L, spectrum, gen, rms=1.0):
    """Real random-phase field with an isotropic shell spectrum (float64)."""
    k = torch.sqrt(_k2(N, L)) * (L / TWO_PI)  # in units of the box mode
    ks = torch.where(k > 0, k, torch.ones_like(k))
    if spectrum == "kminus3":
        shell = ks**-3.0
    elif spectrum == "k0_8":
        shell = (ks / 8) ** 4 * torch.exp(-2 * (ks / 8) ** 2)
    else:
        shell = ks**4 * torch.exp(-((ks / min(10.0, N / 6.0)) ** 2))
    amp = torch.sqrt(shell / (TWO_PI * ks))
    amp[0, 0] = 0.0
    ph = torch.rand((N, N), generator=gen, device="cuda", dtype=torch.float64) * TWO_PI
    f = torch.fft.ifft2(torch.polar(amp, ph)).real
    return f * (rms / torch.sqrt((f * f).mean()))


def _blob(N, L, cx, cy, width):
    x = torch.arange(N, device="cuda", dtype=torch.float64) * (L / N)
    s = L / TWO_PI

    def d(x, c):
        return torch.remainder(x - c * s + L / 2, L) - L / 2

    return torch.exp(-(d(x, cx)[:, None] ** 2 + d(x, cy)[None, :] ** 2) / (2 * (width * s) ** 2))


def _flow_fields(case, seed):
    """theta and the scalars in physical space (plan precision)."""
    N, L, gen = case["N"], case["L"], _gen(seed)
    if case["spectrum"] == "sines":
        x = torch.arange(N, device="cuda", dtype=torch.float64) * (L / N)
        th = torch.sin(4 * x)[:, None] * torch.cos(4 * x)[None, :]
        th = th + 1e-3 * torch.randn((N, N), generator=gen, device="cuda", dtype=torch.float64)
    else:
        th = _random_field(N, L, case["spectrum"], gen)
    scal = [_blob(N, L, 2.0 + i, 3.0, 0.3) + _random_field(N, L, "kminus3", gen, 0.1) for i in range(case["scalars"])]
    return [f.to(_rdtype(case)) for f in [th] + scal]


def _running(case, f):
    """The spectrum of a run in progress: f's modes inside the dealiasing disk."""
    fh = torch.fft.fft2(f.to(torch.float64)) * _mask(case["N"], case["L"])
    return fh.to(C128 if case["precision"] == "float64" else torch.complex64)


def _phases(n_steps, n_ring, seed):
    return torch.rand((n_steps, n_ring), generator=_gen(seed + 1), device="cuda", dtype=torch.float64) * TWO_PI


def _flow_objects(case):
    g = P.make_grid(case["N"], case["L"])
    ring = P.RingForcing(case["kf"], case["dk"], case["eps"]) if case["kf"] > 0 else None
    damp = P.CombinedDamping(case["mu"], max(case["kf"], 4.0), case["nu"], case["p"])
    if case["nu"] == 0 and case["mu"] == 0:
        damp = None
    kw = dict(precision=case["precision"], scheme=case["scheme"])
    if case["kind"] == "rhs":
        return g, None, None, P.gSQGSolver(g, case["alpha"], case["nu"], case["p"], **kw)
    if case["scalars"]:
        sp = {f"c{i}": {"kappa": case["kappa"], "source": P.MeanGradientSource(1.0, 0.0) if case["source"] else None}
              for i in range(case["scalars"])}
        return g, ring, damp, P.gSQGSolverWithScalars(g, case["alpha"], 0.0, case["p"], passive_scalars=sp, **kw)
    return g, ring, damp, P.gSQGSolver(g, case["alpha"], 0.0, case["p"], **kw)


def _sizes(case):
    return [N for N in (32, 64, 128, 256, 512) if f"n{N}" in case]


def _layout(case):
    """(N, alpha, scalar count) of every member, fixed by the case."""
    rng = np.random.default_rng(case["layout"])
    return [(N, float(rng.choice([0.0, 0.5, 1.0, 1.5])), int(rng.integers(0, 4)))
            for N in _sizes(case) for _ in range(case[f"n{N}"])]


def _ensemble_fields(case, seed):
    gen, out = _gen(seed), []
    for N, _, ns in _layout(case):
        c = torch.rand((max(ns, 1), 2), generator=gen, device="cuda", dtype=torch.float64) * TWO_PI
        out.append([_random_field(N, TWO_PI, "k0_8", gen)] + [_blob(N, TWO_PI, c[q, 0], c[q, 1], 0.3) for q in range(ns)])
    return [[f.to(_rdtype(case)) for f in m] for m in out]


def _weights(seed):
    """He-scaled random weights in the network's layout (tap-major)."""
    gen, out = _gen(seed + 2), {}
    for i in range(1, 7):
        shape = (9, 64, 64) if 1 < i < 6 else (9, 64)
        w = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
        out[f"w{i}"] = (w * math.sqrt(2.0 / (9 if i == 1 else 576))).float()
        out[f"b{i}"] = torch.zeros(1 if i == 6 else 64, device="cuda")
    return out


def _train_batch(case, seed):
    n, b, gen = case["size"], case["batch"], _gen(seed)
    x = torch.stack([_random_field(n, TWO_PI, "kminus3", gen) for _ in range(b)])
    t = torch.stack([_random_field(n, TWO_PI, "k4exp", gen) for _ in range(b)])
    return x.float(), t.float()


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "ensemble":
        fields = _ensemble_fields(case, seed)
        members = [Member(N, a, f[0], f[1:], [1e-4] * ns) for (N, a, ns), f in zip(_layout(case), fields)]
        s["solver"] = EnsembleSolver(members, nu_p=case["nu"], p=case["p"], precision=case["precision"])
        return s
    if kind == "closure_train":
        s["net"] = ClosureCNN(case["size"], case["size"], max_batch=case["batch"])
        s["net"].load_state_dict(_weights(seed))
        s["x"], s["t"] = _train_batch(case, seed)
        return s
    if kind == "closure_solve":
        g = P.make_grid(case["N"], case["L"])
        ring = P.RingForcing(case["kf"], case["dk"], case["eps"])
        damp = P.CombinedDamping(case["mu"], case["kf"], case["nu"], case["p"])
        solver = P.gSQGSolver(g, case["alpha"], 0.0, case["p"], precision=case["precision"], scheme="ifrk4")
        s["solver"] = ClosureSolver(solver, SubgridClosure.load(WEIGHTS), damp, ring, forcing_substeps=case["substeps"])
        s["state"] = {"theta_hat": _closure_theta(case, seed), "time": 0.0, "step": 0}
        s["noise"] = _phases(case["steps"] * case["substeps"], s["solver"].n_ring, seed)
        return s
    g, ring, damp, solver = _flow_objects(case)
    fields = _flow_fields(case, seed)
    s.update(grid=g, ring=ring, damp=damp, solver=solver)
    if kind == "transforms":
        s["field"] = fields[0]
        return s
    if kind != "rhs":
        solver.plan(damp, ring)
    if case["start"] == "running":
        st = {"theta_hat": _running(case, fields[0]), "time": 0.0, "step": 0}
        if case["scalars"]:
            st["scalar_state"] = P.MultiScalarState(
                scalars={f"c{i}": _running(case, f) for i, f in enumerate(fields[1:])}, time=0.0, diagnostics={})
    elif case["scalars"]:
        st = solver.initialize(theta0=fields[0], scalar_init={f"c{i}": f for i, f in enumerate(fields[1:])})
    else:
        st = solver.initialize(theta0=fields[0])
    s["state"] = st
    if ring is not None:
        s["noise"] = _phases(case["steps"], ring.n_modes(g), seed)
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------


def _gather(case, thetas, scalars):
    """One tensor per size class: the thetas of its members, then their
    scalars, as an output of the run collects them."""
    out = {N: [] for N in _sizes(case)}
    for th in thetas:
        out[th.shape[0]].append(th)
    for sc in scalars:
        for t in sc:
            out[t.shape[0]].append(t)
    return [torch.stack(v) for v in out.values()]


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "step":
        ring = s["ring"]
        forcing = None if ring is None else ring.bind(s["noise"][0], case["dt"], s["grid"])
        st = s["solver"].step(s["state"], case["dt"], forcing=forcing, damping=s["damp"])
        if case["scalars"]:
            return [st["theta_hat"]] + list(st["scalar_state"].scalars.values())
        return [st["theta_hat"]]
    if kind == "multistep":
        st = s["solver"].multistep(s["state"], case["steps"], case["dt"], forcing=s["ring"], damping=s["damp"],
                                   noise=s.get("noise"))
        return [st["theta_hat"]]
    if kind == "rhs":
        return [s["solver"].compute_rhs(s["state"]["theta_hat"])]
    if kind == "transforms":
        st = s["solver"].initialize(theta0=s["field"])
        u, v = s["solver"].compute_velocity(st["theta_hat"])
        return [st["theta_hat"], u, v]
    if kind == "ensemble":
        e = s["solver"]
        e.multistep(case["steps"], case["dt"])
        return _gather(case, e.theta, e.scalars)
    if kind == "closure_solve":
        return [s["solver"].multistep(s["state"], case["steps"], case["dt"], s["noise"])["theta_hat"]]
    loss = s["net"].train_step(s["x"], s["t"])
    return [loss, s["net"].grad]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------


def _fft_flops(N):
    return 2.5 * N * N * math.log2(N * N)  # one real 2-D transform


def work(case):
    """Bytes: inputs once, outputs once.  Flops: the real 2-D transforms (five
    per right-hand side of theta, three per scalar's, two for a velocity), or
    the convolutions of the network."""
    kind = case["kind"]
    if kind == "closure_train":
        n, b = case["size"], case["batch"]
        mac = b * n * n * (4 * 9 * 64 * 64 + 2 * 9 * 64)
        params = 2 * (9 * 64) + 4 * (9 * 64 * 64 + 64) + 65
        return {"bytes": 2 * b * n * n * 4 + 8 * params * 4, "flops": 2 * 3 * mac}
    cs = 16 if case["precision"] == "float64" else 8
    if kind == "ensemble":
        by = fl = 0
        for N, _, ns in _layout(case):
            by += 2 * cs * N * N * (1 + ns)
            fl += case["steps"] * _fft_flops(N) * (20 + 12 * ns + (2 if ns else 0))
        return {"bytes": by, "flops": fl}
    N = case["N"]
    if kind == "closure_solve":
        conv = 2 * N * N * (4 * 9 * 64 * 64 + 2 * 9 * 64)
        return {"bytes": 2 * cs * N * N, "flops": case["steps"] * 4 * (conv + 6 * _fft_flops(N))}
    if kind == "rhs":
        return {"bytes": 2 * cs * N * N, "flops": 5 * _fft_flops(N)}
    if kind == "transforms":
        return {"bytes": (cs // 2 + cs + cs) * N * N, "flops": 3 * _fft_flops(N)}
    ns = case["scalars"]
    return {"bytes": 2 * cs * N * N * (1 + ns),
            "flops": case["steps"] * _fft_flops(N) * (20 + 12 * ns + (2 if ns else 0))}


# ---------------------------------------------------------------------------
# The same outputs in float64 from plain torch
# ---------------------------------------------------------------------------


def _mask(N, L):
    return torch.sqrt(_k2(N, L)) < (2.0 / 3.0) * (np.pi * N / L)


def _real_ifft(f):
    return torch.fft.ifft2(f).real


class _Spectral:
    """Operators of one grid on (..., N, N) complex128 spectra."""

    def __init__(self, N, L):
        k = _k1d(N, L)
        self.kx, self.ky = k[:, None].expand(N, N), k[None, :].expand(N, N)
        self.k2 = _k2(N, L)
        self.mask = _mask(N, L)

    def velocity(self, th, alpha):
        inv = torch.where(self.k2 > 0, torch.sqrt(torch.where(self.k2 > 0, self.k2, 1.0)) ** (-alpha), 0.0)
        psi = inv * th
        return _real_ifft(-1j * self.ky * psi), _real_ifft(1j * self.kx * psi)

    def advect(self, sh, u, v, extra=None):
        j = u * _real_ifft(1j * self.kx * sh)
        j = j + v * _real_ifft(1j * self.ky * sh)
        if extra is not None:
            j = j - extra
        return -torch.fft.fft2(j.to(C128)) * self.mask

    def drag(self, mu, kf):
        return mu * (torch.sqrt(self.k2) < kf / 2)

    def viscous(self, nu, p):
        return nu * self.k2 ** (p / 2)


def _rk4(th, rhs, dt):
    k = rhs(th)
    acc = th + dt / 6 * k
    k = rhs(th + dt / 2 * k)
    acc += dt / 3 * k
    k = rhs(th + dt / 2 * k)
    acc += dt / 3 * k
    return acc + dt / 6 * rhs(th + dt * k)


def _ifrk4(th, nl, lin, dt):
    e = torch.exp(lin * (dt / 2))
    k1 = nl(th)
    k2 = nl(e * (th + dt / 2 * k1))
    acc = e * e * (th + dt / 6 * k1)
    del k1
    k3 = nl(e * th + dt / 2 * k2)
    acc += dt / 3 * e * (k2 + k3)
    return acc + dt / 6 * nl(e * e * th + dt * e * k3)


def _ring_force(sp, case, phases):
    ring = torch.abs(torch.sqrt(sp.k2) - case["kf"]) <= case["dk"] / 2
    raw = torch.zeros(sp.k2.shape, dtype=C128, device="cuda")
    raw[ring] = torch.polar(torch.full_like(phases, math.sqrt(case["eps"])), phases)
    N = raw.shape[0]
    for i, j in ((0, 0), (N // 2, 0), (0, N // 2), (N // 2, N // 2)):
        raw[i, j] = raw[i, j].real.clone()
    phys = _real_ifft(raw)

    def force(th):
        rate = float((_real_ifft(th) * phys).mean())
        return raw * (case["eps"] / rate if abs(rate) > 1e-10 else 1.0)

    return force


def _exact_flow(case, seed):
    N, L, dt, alpha = case["N"], case["L"], case["dt"], case["alpha"]
    sp = _Spectral(N, L)
    fields = _flow_fields(case, seed)
    if case["kind"] == "transforms":
        th = torch.fft.fft2(fields[0].to(torch.float64))
        return [th, *sp.velocity(th, alpha)]
    if case["start"] == "running":
        spec = [_running(case, f).to(C128) for f in fields]
    else:
        spec = [torch.fft.fft2(f.to(torch.float64)) for f in fields]
    th, scal = spec[0], spec[1:]
    explicit = case["scheme"] == "explicit"
    visc = sp.viscous(case["nu"], case["p"])
    if case["kind"] == "rhs":
        return [sp.advect(th, *sp.velocity(th, alpha)) - visc * th]
    lin = -visc - sp.drag(case["mu"], max(case["kf"], 4.0))
    ring = case["kf"] > 0
    noise = _phases(case["steps"], int((torch.abs(torch.sqrt(sp.k2) - case["kf"]) <= case["dk"] / 2).sum()), seed)
    for n in range(case["steps"]):
        force = _ring_force(sp, case, noise[n]) if ring else None

        def nl(t):
            r = sp.advect(t, *sp.velocity(t, alpha))
            return r if force is None else r + force(t)

        th = _rk4(th, lambda t: nl(t) + lin * t, dt) if explicit else _ifrk4(th, nl, lin, dt)
    if scal:
        u, v = sp.velocity(th, alpha)
        src = -torch.fft.fft2(u.to(C128)) if case["source"] else 0.0
        lin = -case["kappa"] * sp.k2
        for i, s0 in enumerate(scal):
            if explicit:
                scal[i] = _rk4(s0, lambda t: sp.advect(t, u, v) + src + lin * t, dt)
            else:
                scal[i] = _ifrk4(s0, lambda t: sp.advect(t, u, v) + src, lin, dt)
    return [th] + scal


def _exact_ensemble(case, seed):
    sps = {N: _Spectral(N, TWO_PI) for N in _sizes(case)}
    thetas, scalars = [], []
    for (N, alpha, ns), fields in zip(_layout(case), _ensemble_fields(case, seed)):
        sp = sps[N]
        th, scal = torch.fft.fft2(fields[0].double()), [torch.fft.fft2(f.double()) for f in fields[1:]]
        lin, dt = -sp.viscous(case["nu"], case["p"]), case["dt"]
        for _ in range(case["steps"]):
            th = _ifrk4(th, lambda t: sp.advect(t, *sp.velocity(t, alpha)), lin, dt)
            if ns:
                u, v = sp.velocity(th, alpha)
                scal = [_ifrk4(t0, lambda t: sp.advect(t, u, v), -1e-4 * sp.k2, dt) for t0 in scal]
        thetas.append(th)
        scalars.append(scal)
    return _gather(case, thetas, scalars)


def _conv(x, w, b):
    return torch.nn.functional.conv2d(torch.nn.functional.pad(x, (1, 1, 1, 1), mode="circular"), w, b)


def _network(p, x):
    """The six-layer network on x [B, H, W] in float64; p as ClosureCNN lays
    its parameters out (tap-major weights)."""
    gelu = torch.nn.functional.gelu
    a = gelu(_conv(x[:, None], p["w1"].t().reshape(64, 1, 3, 3), p["b1"]), approximate="tanh")
    for i in range(2, 6):
        w = p[f"w{i}"].permute(1, 2, 0).reshape(64, 64, 3, 3)
        a = gelu(_conv(a, w, p[f"b{i}"]), approximate="tanh")
    return _conv(a, p["w6"].t().reshape(1, 64, 3, 3), p["b6"])[:, 0]


def _exact_train(case, seed):
    p = {k: w.double().requires_grad_() for k, w in _weights(seed).items()}
    x, t = (f.double() for f in _train_batch(case, seed))
    loss = 0.0
    for i in range(case["batch"]):  # one sample at a time: float64 activations are large
        part = ((_network(p, x[i:i + 1]) - t[i:i + 1]) ** 2).sum() / t.numel()
        part.backward()
        loss += float(part.detach())
    return [torch.tensor(loss, dtype=torch.float64), torch.cat([g.grad.reshape(-1) for g in p.values()])]


def _closure_theta(case, seed):
    """A coarse state of a running solve: random phases inside the disk."""
    f = _random_field(case["N"], case["L"], "k4exp", _gen(seed))
    return (torch.fft.fft2(f) * _mask(case["N"], case["L"])).to(torch.complex64)


def _exact_closure_solve(case, seed):
    sp, dt, m = _Spectral(case["N"], case["L"]), case["dt"], case["substeps"]
    z = np.load(WEIGHTS)
    p = {n: torch.as_tensor(z[n], device="cuda").double() for n in z.files if n[0] in "wb"}
    st, sx = float(z["sigma_theta"]), float(z["sigma_pi"])
    th = _closure_theta(case, seed).to(C128)
    lin = -sp.viscous(case["nu"], case["p"]) - sp.drag(case["mu"], case["kf"])
    n_ring = int((torch.abs(torch.sqrt(sp.k2) - case["kf"]) <= case["dk"] / 2).sum())
    noise = _phases(case["steps"] * m, n_ring, seed)

    def nl(t):
        pi = _network(p, _real_ifft(t)[None] / st)[0] * sx
        return sp.advect(t, *sp.velocity(t, case["alpha"]), extra=pi)

    with torch.no_grad():
        for n in range(case["steps"]):
            rows = [_ring_force(sp, case, noise[n * m + i]) for i in range(m)]
            for f in rows[:m // 2]:
                th = _rk4(th, f, dt / m)
            th = _ifrk4(th, nl, lin, dt)
            for f in rows[m // 2:]:
                th = _rk4(th, f, dt / m)
    return [th]


def exact(case, seed):
    return {"ensemble": _exact_ensemble, "closure_train": _exact_train,
            "closure_solve": _exact_closure_solve}.get(case["kind"], _exact_flow)(case, seed)
