"""Spectra with and without modes outside the dealiasing band, where the passes
leave rows and modes out: each form against the float64 oracle (<= 1e-12
relative L2 in double, 2e-5 in single precision, the bars of the other parity
tests)."""

import numpy as np
import pytest
import torch

from oracle import sqg_oracle as O

pytestmark = pytest.mark.gpu

TWO_PI = 2 * np.pi
TOL = {"float64": 1e-12, "float32": 2e-5}


@pytest.fixture(scope="module")
def P():
    from pygsquig_b200.build import build

    build()
    import pygsquig_b200 as P

    return P


def rel(a, b):
    return float(np.linalg.norm(a.detach().cpu().numpy() - b) / max(np.linalg.norm(b), 1e-300))


def spectrum(N, form, seed):
    """A field's spectrum: full; inside the band; rows just beyond it; one
    conjugate pair far beyond it."""
    k = np.abs(np.fft.fftfreq(N, 1.0 / N))
    r = np.sqrt(k[:, None] ** 2 + k[None, :] ** 2)
    fh = np.fft.fft2(np.random.default_rng(seed).standard_normal((N, N))) / (1 + r) ** 2
    if form == "rows":
        fh = fh * (k[:, None] < N / 3 + 2)
    elif form != "full":
        fh = fh * (r < N / 3)
    if form == "pair":
        fh[N // 2 - 1, 1], fh[N // 2 + 1, N - 1] = 0.3 + 0.2j, 0.3 - 0.2j
    return fh


@pytest.mark.parametrize("form", ["full", "band", "rows", "pair"])
@pytest.mark.parametrize("N,prec", [(8, "float64"), (32, "float32"), (64, "float64"), (512, "float64"),
                                    (1024, "float32")])
@pytest.mark.parametrize("scheme", ["ifrk4", "explicit"])
def test_step_with_scalars(P, N, prec, form, scheme):
    dt, nu = 1e-3, 0.3 / (N / 3.0) ** 4 / 1e-3  # nu k^4 dt = 0.3 at the band's edge (1.5 at the corner: stable)
    th, sa, sb = spectrum(N, form, 1), spectrum(N, "band", 2), spectrum(N, form, 3)
    g, go = P.make_grid(N, TWO_PI), O.make_grid(N, TWO_PI)
    s = P.gSQGSolverWithScalars(g, 0.5, nu, 4, precision=prec, scheme=scheme, passive_scalars={
        "a": {"kappa": 1e-3, "source": P.MeanGradientSource(1.0, 0.5)}, "b": {"kappa": 1e-3}})
    so = O.gSQGSolverWithScalars(go, 0.5, nu, 4, scheme=scheme, passive_scalars={
        "a": {"kappa": 1e-3, "source": O.MeanGradientSource(1.0, 0.5)}, "b": {"kappa": 1e-3, "source": None}})
    cdt = torch.complex128 if prec == "float64" else torch.complex64
    t = lambda x: torch.as_tensor(x).to("cuda", cdt)  # noqa: E731
    st = {"theta_hat": t(th), "time": 0.0, "step": 0,
          "scalar_state": P.MultiScalarState({"a": t(sa), "b": t(sb)}, 0.0, {})}
    ro = {"theta_hat": th, "time": 0.0, "step": 0, "scalars": {"a": sa, "b": sb}}
    for _ in range(2):
        st, ro = s.step(st, dt), so.step(ro, dt)
    assert rel(st["theta_hat"], ro["theta_hat"]) < TOL[prec]
    for q in "ab":
        assert rel(st["scalar_state"].scalars[q], ro["scalars"][q]) < TOL[prec]
    # several steps in one call: the flags are carried from step to step
    s1 = P.gSQGSolver(g, 0.5, nu, 4, precision=prec, scheme=scheme)
    m = s1.multistep({"theta_hat": t(th), "time": 0.0, "step": 0}, 2, dt)
    assert rel(m["theta_hat"], ro["theta_hat"]) < TOL[prec]
    assert rel(s1.compute_rhs(t(th)), so.compute_rhs(th)) < TOL[prec]
    u, v = s1.compute_velocity(t(th))
    uo, vo = so.compute_velocity(th)
    assert max(rel(u, uo), rel(v, vo)) < TOL[prec]


@pytest.mark.parametrize("N", [64, 512])
def test_terms_that_reach_outside(P, N):
    """A callable term on every mode, and a forced ring outside the band."""
    th = spectrum(N, "band", 5)
    g, go = P.make_grid(N, TWO_PI), O.make_grid(N, TWO_PI)
    s, so = P.gSQGSolver(g, 1.0), O.gSQGSolver(go, 1.0)
    st = {"theta_hat": torch.as_tensor(th).cuda(), "time": 0.0, "step": 0}
    out = s.step(st, 1e-3, forcing=lambda x: 0.1 * x + 0.05)
    ref = so.step({"theta_hat": th, "time": 0.0, "step": 0}, 1e-3, forcing=lambda x: 0.1 * x + 0.05)
    assert rel(out["theta_hat"], ref["theta_hat"]) < 1e-12
    kf = N / 2.0 - 3
    th = th + 1e-3 * spectrum(N, "full", 6)  # an overlap with the ring, so that its rescale is well conditioned
    ring, ro = P.RingForcing(kf, 2.0, 0.1), O.RingForcing(kf, 2.0, 0.1)
    ph = np.angle(th[np.asarray(ro.get_forcing_mask(go))])
    st["theta_hat"] = torch.as_tensor(th).cuda()
    out = s.step(st, 1e-4, forcing=ring.bind(ph, 1e-4, g))
    ref = O.step_forced(so, {"theta_hat": th, "time": 0.0, "step": 0}, 1e-4, ro, ph, None)
    assert rel(out["theta_hat"], ref["theta_hat"]) < 1e-12


@pytest.mark.parametrize("N", [16, 256, 1024])
@pytest.mark.parametrize("prec", ["float64", "float32"])
def test_real_fields_at_any_element(P, N, prec):
    """Real fields that start on one element's alignment take the same values."""
    from pygsquig_b200._plan import PlanKey, get_plan

    pl = get_plan(PlanKey(N=N, L=TWO_PI, alpha=1.0, nu_p=0.0, p=8, precision=prec))
    f = torch.randn(N, N, device="cuda", dtype=pl.rdtype)
    odd = torch.empty(N * N + 1, device="cuda", dtype=pl.rdtype)[1:].view(N, N)
    odd.copy_(f)
    fh = pl.to_spectral(f)
    assert torch.equal(pl.to_spectral(odd), fh)
    assert torch.equal(pl.to_physical(fh, out=odd), pl.to_physical(fh))


def stage_setup(P, N, prec, scheme, nu):
    """A plan whose workspace holds another field's values at every mode, a
    band-limited state and the oracle."""
    g, go = P.make_grid(N, TWO_PI), O.make_grid(N, TWO_PI)
    s = P.gSQGSolver(g, 1.0, nu, 4, precision=prec, scheme=scheme)
    so = O.gSQGSolver(go, 1.0, nu, 4, scheme=scheme)
    pl = s.plan()
    dt = torch.complex128 if prec == "float64" else torch.complex64
    other = torch.as_tensor(spectrum(N, "full", 8)).to("cuda", dt)
    pl.step(other, torch.empty_like(other), 1e-3)
    th = spectrum(N, "band", 9)
    return pl, so, go, th, torch.as_tensor(th).to("cuda", dt)


@pytest.mark.parametrize("N,prec", [(512, "float64"), (1024, "float32")])
@pytest.mark.parametrize("scheme", ["ifrk4", "explicit"])
@pytest.mark.parametrize("given", ["-f-f", "--f-", "---f", "p-f-", "pfpp"])
def test_terms_at_some_stages_only(P, N, prec, scheme, given):
    """Stage by stage: a spectral term (f), a physical one (p) or none (-)."""
    dt = 1e-3
    pl, so, go, th, t0 = stage_setup(P, N, prec, scheme, 0.3 / (N / 3.0) ** 4 / dt)
    src = np.random.default_rng(3).standard_normal((N, N))
    terms = {"f": 100.0 * spectrum(N, "full", 7), "p": go.dealias_mask * np.fft.fft2(src), "-": np.zeros((N, N))}
    fd, pd = torch.as_tensor(terms["f"]).to(t0), torch.as_tensor(src).to("cuda", pl.rdtype)
    out = torch.empty_like(t0)
    pl.stage_begin(t0)
    for s, k in enumerate(given, 1):
        if k == "p":
            pl.stage_physical(s, t0, out, dt, pd)
        else:
            pl.stage(s, t0, out, dt, fd if k == "f" else None)
    order = iter(given)
    ref = so.step({"theta_hat": th, "time": 0.0, "step": 0}, dt, forcing=lambda x: terms[next(order)])["theta_hat"]
    assert rel(out, ref) < TOL[prec]


@pytest.mark.parametrize("N,prec", [(512, "float64"), (1024, "float32")])
def test_stage_buffer_of_a_whole_step(P, N, prec):
    """The buffer holds the last stage's input at every mode after a step whose
    stages store it (explicit scheme with a linear term)."""
    from pygsquig_b200 import _lib

    dt = 1e-3
    pl, so, go, th, t0 = stage_setup(P, N, prec, "explicit", 0.3 / (N / 3.0) ** 4 / dt)
    pl.step(t0, torch.empty_like(t0), dt)
    x = th
    for f in (0.5, 0.5, 1.0):
        x = th + f * dt * so.compute_rhs(x)
    buf = pl.buffer(_lib.SQG_BUF_STAGE, t0.dtype, t0.shape)
    assert rel(buf, x) < TOL[prec]
    k = np.abs(np.fft.fftfreq(N, 1.0 / N))
    outside = torch.as_tensor(k[:, None] ** 2 + k[None, :] ** 2 > (N / 3.0 + 1) ** 2, device="cuda")
    assert torch.count_nonzero(buf[outside]) == 0


@pytest.mark.parametrize("N,prec", [(512, "float64"), (1024, "float32")])
@pytest.mark.parametrize("p", [0, 3, 170, 171, -1])
def test_one_mode_outside_at_every_element(P, N, prec, p):
    """A row's flag sees one non-zero mode outside the band at whichever element it
    stands (a single wave advects nothing: it stays as it is)."""
    p = p % (N // 2 + 1)
    s = P.gSQGSolver(P.make_grid(N, TWO_PI), 1.0, 0.0, 4, precision=prec, scheme="ifrk4")
    pl = s.plan()
    th = torch.zeros(N, N, dtype=pl.cdtype, device="cuda")
    out = torch.empty_like(th)
    worst = torch.zeros((), device="cuda", dtype=pl.rdtype)
    for iy in range(N):
        ky = min(iy, N - iy)
        if p * p + ky * ky <= (N / 3.0 + 1) ** 2 or (p % (N // 2) == 0 and ky % (N // 2) == 0):
            continue
        th.zero_()
        th[p, iy], th[-p % N, -iy % N] = 1 + 2j, 1 - 2j
        pl.step(th, out, 1e-3)
        worst = torch.maximum(worst, (out - th).abs().max())
    assert float(worst) < 5 * TOL[prec]


@pytest.mark.parametrize("prec", ["float64", "float32"])
def test_smallest_ensemble_with_modes_outside(P, prec):
    """N = 8: one transform pass, several warps to a block.  Members that hold one
    mode outside the band each, against the single field's passes (every mode)."""
    from pygsquig_b200.ensemble import EnsembleSolver, Member

    N, modes = 8, [(p, iy) for p in range(5) for iy in range(8) if p * p + min(iy, 8 - iy) ** 2 >= 8]
    z = np.zeros((N, N))
    e = EnsembleSolver([Member(N, 1.0, z, [z], [1e-3]) for _ in modes], nu_p=1e-6, p=8, precision=prec)
    band = spectrum(N, "band", 4)
    solver = P.gSQGSolver(P.make_grid(N, TWO_PI), 1.0, 1e-6, 8, precision=prec, scheme="ifrk4")
    ref = []
    for i, (p, iy) in enumerate(modes):
        th = band.copy()
        th[p, iy], th[-p % N, -iy % N] = 0.3 + 0.2j, 0.3 - 0.2j
        e.theta[i].copy_(torch.as_tensor(th))
        e.scalars[i][0].copy_(torch.as_tensor(th))
        st = {"theta_hat": e.theta[i].clone(), "time": 0.0, "step": 0}
        ref.append(solver.multistep(st, 2, 1e-3)["theta_hat"])
    e.multistep(2, 1e-3)
    for a, b in zip(e.theta, ref):
        assert rel(a, b.cpu().numpy()) < TOL[prec]
    for i, (p, iy) in enumerate(modes):  # a scalar's mode outside decays by diffusion alone
        if p % 4 == 0 and iy % 4 == 0:
            continue  # its own conjugate
        k2 = p * p + min(iy, N - iy) ** 2
        assert abs(complex(e.scalars[i][0][p, iy].item()) / (0.3 + 0.2j) - np.exp(-2e-6 * k2)) < TOL[prec]


def rows_of(N, form, seed):
    """As spectrum(); "mixed": of the rows beyond the band every fifth is held."""
    if form != "mixed":
        return spectrum(N, form, seed)
    k = np.abs(np.fft.fftfreq(N, 1.0 / N))
    keep = (k[:, None] <= N // 3) | (k[:, None] % 5 == 0)
    return spectrum(N, "full", seed) * keep


@pytest.fixture(scope="module")
def threaded():
    """The oracle's transforms on several threads (large grids)."""
    O.set_fft_workers(16)
    yield
    O.set_fft_workers(1)


@pytest.mark.parametrize("N", [2048, 4096])
@pytest.mark.parametrize("form,other", [("rows", "mixed"), ("pair", "band"), ("mixed", "pair"), ("band", "full")])
def test_large_step_with_some_rows_held(P, threaded, N, form, other):
    """A step with a scalar whose rows differ from theta's: at these sizes the
    rows beyond the band arrive in fetches of their own."""
    dt = 1e-3
    nu = 0.3 / (N / 3.0) ** 4 / dt
    g, th, sa = P.make_grid(N, TWO_PI), rows_of(N, form, 1), rows_of(N, other, 3)
    so = O.gSQGSolverWithScalars(O.make_grid(N, TWO_PI), 0.5, nu, 4, scheme="ifrk4", passive_scalars={
        "a": {"kappa": 1e-3, "source": O.MeanGradientSource(1.0, 0.5)}})
    ref = so.step({"theta_hat": th, "time": 0.0, "step": 0, "scalars": {"a": sa}}, dt)
    for prec, cdt in (("float64", torch.complex128), ("float32", torch.complex64)):
        s = P.gSQGSolverWithScalars(g, 0.5, nu, 4, precision=prec, scheme="ifrk4", passive_scalars={
            "a": {"kappa": 1e-3, "source": P.MeanGradientSource(1.0, 0.5)}})
        t, q = (torch.as_tensor(x).to("cuda", cdt) for x in (th, sa))
        st = s.step({"theta_hat": t, "time": 0.0, "step": 0, "scalar_state": P.MultiScalarState({"a": q}, 0.0, {})}, dt)
        assert rel(st["theta_hat"], ref["theta_hat"]) < TOL[prec]
        assert rel(st["scalar_state"].scalars["a"], ref["scalars"]["a"]) < TOL[prec]
        # from the second step on, the last stage sets the flags of the next
        s1 = P.gSQGSolver(g, 0.5, nu, 4, precision=prec, scheme="ifrk4")
        x = {"theta_hat": t, "time": 0.0, "step": 0}
        two = s1.step(s1.step(x, dt), dt)["theta_hat"].cpu().numpy()
        assert rel(s1.multistep(x, 2, dt)["theta_hat"], two) < TOL[prec]


@pytest.mark.parametrize("form", ["rows", "pair", "mixed", "band"])
@pytest.mark.parametrize("N", [2048, 4096])
def test_large_rhs_and_velocity_with_some_rows_held(P, threaded, N, form):
    th, go = rows_of(N, form, 1), O.make_grid(N, TWO_PI)
    so = O.gSQGSolver(go, 0.5, 1e-8, 2)
    rhs, vel = so.compute_rhs(th), so.compute_velocity(th)
    for prec in ("float64", "float32"):
        s = P.gSQGSolver(P.make_grid(N, TWO_PI), 0.5, 1e-8, 2, precision=prec)
        t = torch.as_tensor(th).cuda()
        assert rel(s.compute_rhs(t), rhs) < TOL[prec]
        for a, b in zip(s.compute_velocity(t), vel):
            assert rel(a, b) < TOL[prec]


@pytest.mark.parametrize("sizes", [(32, 64), (128, 512), (256, 1024)])
@pytest.mark.parametrize("prec", ["float64", "float32"])
def test_ensemble_members_with_some_rows_held(P, sizes, prec):
    """Theta and scalars hold different rows: the unified passes (128, 512) and
    the passes class by class."""
    from pygsquig_b200.ensemble import EnsembleSolver, Member

    forms = [("band", "full"), ("full", "band"), ("pair", "rows"), ("mixed", "pair"), ("band", "band")]
    members = [(N, f) for N in sizes for f in (forms if N < 1024 else forms[2:4])]
    nu, dt = 0.3 / (max(sizes) / 3.0) ** 8 / 1e-3, 1e-3
    e = EnsembleSolver([Member(N, 0.5, np.zeros((N, N)), [np.zeros((N, N))] * 2, [1e-3, 1e-4]) for N, _ in members],
                       nu_p=nu, p=8, precision=prec)
    refs = []
    for i, (N, (a, b)) in enumerate(members):
        th, s1, s2 = rows_of(N, a, i), rows_of(N, b, 40 + i), rows_of(N, a, 80 + i)
        for t, x in zip([e.theta[i]] + e.scalars[i], (th, s1, s2)):
            t.copy_(torch.as_tensor(x))
        so = O.gSQGSolverWithScalars(O.make_grid(N, TWO_PI), 0.5, nu, 8, scheme="ifrk4", passive_scalars={
            "a": {"kappa": 1e-3, "source": None}, "b": {"kappa": 1e-4, "source": None}})
        st = {"theta_hat": th, "time": 0.0, "step": 0, "scalars": {"a": s1, "b": s2}}
        for _ in range(2):
            st = so.step(st, dt)
        refs.append([st["theta_hat"], st["scalars"]["a"], st["scalars"]["b"]])
    e.multistep(2, dt)
    for i, ref in enumerate(refs):
        for t, x in zip([e.theta[i]] + e.scalars[i], ref):
            assert rel(t, x) < TOL[prec], (members[i], i)
