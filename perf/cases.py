"""Timed cases of the correlated-k forward model with its Jacobian and of the
optimal-estimation step, through the package's public entry points.

The atmospheres, k-tables and CIA table are the seeded synthetic ones of
``radtrancode_b200.synth`` (lognormal k-distributions, a nadir giant-planet
atmosphere): their shapes and distributions are those of the repository's own
configurations.  A run's k-tables stay the same for every seed (they are files
that a user's program loads once); the atmosphere, state and measurement
change with the seed.

``exact`` restates the same physics in 64 bits with plain torch and numpy.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from radtrancode_b200 import cirsradg, synth

ABSORBERS = synth.ABSORBERS_C2
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # one wavenumber of a small atmosphere: the per-wavenumber entry, where latency is all there is
        dict(name="one_wavenumber", kind="wave", nlayer=40, nwave=1, ngas=2, ng=20, angle=0.0),
        # the smallest configuration: one absorber, so no overlap is sorted
        dict(name="small_ch4", kind="spectrum", nlayer=40, nwave=100, ngas=1, ng=20, angle=0.0, dust=0, fwhm=0.0, iform=0),
        # an off-nadir spectrum on 10-point k-tables, the other size these tables are distributed in
        dict(name="ten_point_tables", kind="spectrum", nlayer=73, nwave=515, ngas=3, ng=10, angle=35.0, dust=0, fwhm=0.0, iform=0),
        # an ordinary spectrum through dust, convolved to instrument channels (FWHM > 0)
        dict(name="dust_channels", kind="spectrum", nlayer=60, nwave=401, ngas=2, ng=20, angle=20.0, dust=2, fwhm=2.5, iform=0),
        # the planet's total flux (iform 3): the kernel instance of the less common options
        dict(name="total_flux", kind="spectrum", nlayer=80, nwave=150, ngas=2, ng=16, angle=0.0, dust=0, fwhm=0.0, iform=3),
        # the full-size spectrum
        dict(name="full_spectrum", kind="spectrum", nlayer=120, nwave=2000, ngas=4, ng=20, angle=0.0, dust=0, fwhm=0.0, iform=0),
        # uneven spectra in one call, as a survey of footprints is processed
        dict(name="uneven_batch", kind="batch", nspec=14, nlayer=110, nwave=700, ngas=4, ng=20),
        # the same atmospheres evaluated again and again: prepared once, launched and read back
        dict(name="resident_batch", kind="resident", nspec=5, nlayer=64, nwave=300, ngas=3, ng=20),
        # the Newton steps of a batch of retrievals, and their cost functions
        dict(name="newton_batch", kind="newton", nret=24, nx=124, ny=2000),
        # the end of a retrieval: gain matrix, averaging kernels, error covariances
        dict(name="final_errors", kind="errors", nx=107, ny=900),
        # a spectrum and its Jacobian rows to channels by the standalone convolution
        dict(name="convolve_rows", kind="conv", nser=45, nwave=1000, nconv=230, fwhm=3.0),
        # whole retrievals, every iteration on the device
        dict(name="retrievals", kind="retrieve", nret=4, nlayer=40, nwave=200, ngas=2, ng=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["wave", "spectrum", "spectrum", "spectrum", "spectrum", "batch", "resident", "newton", "errors",
                       "conv", "retrieve"])
    ng = rng.choice([20, 20, 20, 10, 16, 13])
    if kind == "wave":
        return dict(kind=kind, nlayer=rng.randint(20, 120), nwave=1, ngas=rng.randint(1, 4), ng=ng, angle=rng.uniform(0, 70))
    if kind == "spectrum":
        dust = rng.choice([0, 0, 0, 1, 2])
        return dict(kind=kind, nlayer=rng.randint(20, 120), nwave=_log_int(rng, 32, 2000), ngas=rng.randint(1, 4), ng=ng,
                    angle=rng.uniform(0, 70), dust=dust, fwhm=rng.choice([0.0, 0.0, 2.0]),
                    iform=rng.choice([0, 0, 0, 3]))
    if kind == "batch":
        return dict(kind=kind, nspec=rng.randint(2, 12), nlayer=rng.randint(40, 110), nwave=_log_int(rng, 200, 700),
                    ngas=rng.randint(1, 4), ng=ng)
    if kind == "resident":
        return dict(kind=kind, nspec=rng.randint(1, 8), nlayer=rng.randint(40, 110), nwave=_log_int(rng, 50, 400),
                    ngas=rng.randint(1, 4), ng=ng)
    if kind == "newton":
        return dict(kind=kind, nret=_log_int(rng, 1, 24), nx=rng.randint(30, 128), ny=_log_int(rng, 200, 2000))
    if kind == "errors":
        return dict(kind=kind, nx=rng.randint(20, 128), ny=_log_int(rng, 200, 1000))
    if kind == "conv":
        return dict(kind=kind, nser=_log_int(rng, 1, 125), nwave=_log_int(rng, 100, 2000), nconv=rng.randint(20, 400),
                    fwhm=rng.uniform(1.0, 6.0))
    return dict(kind=kind, nret=rng.randint(1, 4), nlayer=rng.randint(30, 50), nwave=rng.randint(100, 250),
                ngas=rng.randint(1, 3), ng=20)


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=6)
def _tables(ng, nbin):
    return synth.make_ktables(ABSORBERS, np_=20, nt=15, ng=ng, vmin=600.0, delv=0.4, nbin=nbin, seed=1002)


def _tables_for(case):
    return _tables(case["ng"], 2000 if case["nwave"] > 500 else 500)


@functools.lru_cache(maxsize=1)
def _cia():
    return synth.make_cia(1002)


def _channels(v0, v1, n, fwhm):
    """n channels inside [v0, v1], away from its ends by more than a width."""
    return synth.Channels(np.linspace(v0 + 1.5 * fwhm, v1 - 1.5 * fwhm, n))


def _spectrum_job(case, seed):
    kt = _tables_for(case)
    rng = np.random.default_rng(seed)
    iw0 = int(rng.integers(0, int(kt.nbin[0]) - case["nwave"] + 1))
    job = synth.make_job(kt, ABSORBERS[:case["ngas"]], nlayer=case["nlayer"], seed=seed, iw0=iw0, nwave=case["nwave"],
                         theta_deg=case.get("angle", 0.0), vmr_perturb=0.3)
    if case.get("dust"):
        job = synth.with_dust(job, case["dust"], seed=seed)
    if case.get("fwhm"):
        ch = _channels(float(job.vwave[0]), float(job.vwave[-1]), max(2, case["nwave"] // 4), case["fwhm"])
        job = dataclasses.replace(job, fwhm=case["fwhm"], conv=ch)
    if case.get("iform"):
        job = dataclasses.replace(job, iform=case["iform"], radius1=71492.0)
    return job


def _batch_jobs(case, seed):
    """Uneven spectra: windows, layer counts, absorbers and angles drawn below the case's largest."""
    kt = _tables_for(case)
    rng = np.random.default_rng(seed)
    jobs = []
    for s in range(case["nspec"]):
        f = (s + 1) / case["nspec"]          # the sizes are the case's own, the same for every seed
        w = max(8, int(case["nwave"] * (0.4 + 0.6 * f)) - (s * 7) % 3)
        L = max(10, int(case["nlayer"] * (1.0 - 0.5 * f)) + (s * 5) % 4)
        na = 1 + s % case["ngas"] if case["nspec"] > 1 else case["ngas"]
        ab = [ABSORBERS[i] for i in sorted(rng.choice(4, size=na, replace=False))]
        jobs.append(synth.make_job(kt, ab, nlayer=L, seed=int(rng.integers(1 << 30)),
                                   iw0=int(rng.integers(0, int(kt.nbin[0]) - w + 1)), nwave=w,
                                   theta_deg=float(rng.uniform(0.0, 70.0)), vmr_perturb=0.3))
    return jobs


def _context(kt=None):
    ctx = cirsradg.Context(0)
    if kt is not None:
        ctx.set_ktables(kt)
        ctx.set_cia(_cia())
    return ctx


def _oe_inputs(nret, nx, ny, seed):
    """Weighting functions in ln p (one gas scale in twelve states), a prior
    covariance and residuals as a retrieval's iterations have them."""
    rng = np.random.default_rng(seed)
    ns = max(1, nx // 31)
    L = nx - ns
    p = np.geomspace(1e6, 10.0, L)
    lnp, v = np.log(p), np.linspace(0.0, 1.0, ny)
    sa = synth.prior_covariance(p, ns)
    sai = np.linalg.inv(sa)
    kk = np.empty((nret, nx, ny), np.float32)
    for r in range(nret):
        c = lnp.min() + (lnp.max() - lnp.min()) * (0.5 + 0.4 * np.sin(9.0 * v + rng.uniform(0, 6)))
        c = c + 0.3 * rng.standard_normal(ny)
        kk[r, :L] = 2e-9 * np.exp(-0.5 * ((lnp[:, None] - c[None, :]) / 1.2) ** 2) * (24.0 / L)
        kk[r, L:] = 1e-8 * np.abs(np.sin(rng.uniform(5, 30, (ns, 1)) * v + rng.uniform(0, 6, (ns, 1))))
    sei = np.full((nret, ny), 1e18) * rng.uniform(0.8, 1.2, (nret, ny))
    xa = np.concatenate([140.0 + 30.0 * np.tanh((lnp - 9.0) / 2.5), np.zeros(ns)])
    ch = np.linalg.cholesky(sa)
    xa = np.repeat(xa[None].astype(np.float32), nret, 0)
    xn = (xa + 0.5 * (ch @ rng.standard_normal((nx, nret))).T).astype(np.float32)
    xt = (xa + (ch @ rng.standard_normal((nx, nret))).T).astype(np.float32)
    yn = (5e-8 + 2e-8 * np.sin(6.0 * v)[None] + np.zeros((nret, 1))).astype(np.float32)
    y = (yn + np.einsum("rij,ri->rj", kk.astype(np.float64), (xt - xn).astype(np.float64))
         + 1e-9 * rng.standard_normal((nret, ny))).astype(np.float32)
    return dict(kk=kk, sei=sei, sa=sa, sai=np.repeat(sai[None], nret, 0), xa=xa, xn=xn, y=y, yn=yn)


def _conv_inputs(case, seed):
    rng = np.random.default_rng(seed)
    v = (600.0 + 0.4 * np.arange(case["nwave"])).astype(np.float32)
    t = np.linspace(0.0, 1.0, case["nwave"])
    y = np.stack([1e-8 * (1.5 + np.sin(rng.uniform(5, 60) * t + rng.uniform(0, 6)) + 0.2 * rng.standard_normal(len(t)))
                  for _ in range(case["nser"])]).astype(np.float32)
    return v, y, _channels(float(v[0]), float(v[-1]), case["nconv"], case["fwhm"])


def _retrieval_cases(case, seed):
    kt = _tables(case["ng"], 500)
    out = []
    for r in range(case["nret"]):
        c = synth.make_retrieval(kt, ABSORBERS[:case["ngas"]], nlayer=case["nlayer"], seed=1000 * seed + 10 * r,
                                 iw0=(37 * r) % (500 - case["nwave"]), nwave=case["nwave"])
        y = _forward64(kt, _cia(), synth.job_at_state(c, c.x_true))[0]   # the measured spectrum
        out.append(synth.observe(c, y, seed=seed + r))
    return kt, out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("wave", "spectrum"):
        job = _spectrum_job(case, seed)
        st = dict(kind=kind, ctx=_context(_tables_for(case)), job=job)
        if kind == "wave":
            st["isw"] = list(range(2, job.ngas + 1))     # the absorbers and the temperature
        return st
    if kind in ("batch", "resident"):
        st = dict(kind=kind, ctx=_context(_tables_for(case)), jobs=_batch_jobs(case, seed))
        if kind == "resident":
            st["ctx"].prepare(st["jobs"])
            st["ctx"].use_graph(True)
        return st
    if kind in ("newton", "errors"):
        return dict(kind=kind, ctx=_context(), **_oe_inputs(case.get("nret", 1), case["nx"], case["ny"], seed))
    if kind == "conv":
        v, y, ch = _conv_inputs(case, seed)
        return dict(kind=kind, ctx=_context(), v=v, y=y, ch=ch, fwhm=case["fwhm"])
    kt, cases = _retrieval_cases(case, seed)
    return dict(kind=kind, ctx=_context(kt), cases=cases)


def run(st):
    ctx, kind = st["ctx"], st["kind"]
    if kind == "wave":
        return ctx.cirsradg_wave(st["job"], st["isw"])
    if kind == "spectrum":
        return ctx.cirsrtfg_wave(st["job"])
    if kind == "batch":
        return ctx.cirsrtfg_wave_batch(st["jobs"])
    if kind == "resident":
        ctx.launch()
        return ctx.fetch()
    if kind == "newton":
        x, nonpd, _ = ctx.newton_step_batch(st["kk"], st["sei"], st["sai"], st["xa"], st["xn"], st["y"], st["yn"])
        phi, chisq = ctx.calc_phiret_batch(st["y"], st["yn"], st["sei"], st["xn"], st["xa"], st["sai"])
        return x, nonpd, phi, chisq
    if kind == "errors":
        dd, aa, nonpd = ctx.calc_gain_matrix(st["kk"][0], st["sai"][0], st["sei"][0])
        x = ctx.calcnextxn(st["xa"][0], st["xn"][0], st["y"][0], st["yn"][0], dd, aa)
        return (x, nonpd, dd, aa) + ctx.calc_serr(st["sa"], 1.0 / st["sei"][0], dd, aa)
    if kind == "conv":
        return ctx.cirsconv_ex(st["v"], st["y"], st["fwhm"], st["ch"])
    return [(r["x"], r["yn"]) for r in ctx.retrieve_batch(st["cases"])]


# -------------------------------------------------------------------- work
def _forward_work(job, ng, nt=15, np_=20):
    """The table cells that the layers touch, the outputs and the inputs once;
    the operations of the overlap (a comparison sort of NG^2 keys and the sums
    of k and of every gradient column per pass) and of the path."""
    na, L, W, n = job.ngas - 2, job.nlayer, job.nwave, ng * ng
    cells = min(4 * L, np_ * nt)
    b = 4.0 * (W * na * cells * ng + job.npath * job.nconv * (job.nv + 2) + W * (2 + na) + L * (8 + 3 * job.ngas)
               + 3 * job.nv)
    passes = float(max(na - 1, 0)) * L * W
    f = passes * n * (3 + math.log2(n) + 2 + 2 * (na + 1)) + float(W) * L * ng * (12 * na + 8 * (na + 2))
    return b, f


def work(case):
    kind = case["kind"]
    if kind in ("wave", "spectrum", "batch", "resident"):
        jobs = [_spectrum_job(case, 1)] if kind in ("wave", "spectrum") else _batch_jobs(case, 1)
        each = [_forward_work(j, case["ng"]) for j in jobs]
        return dict(bytes=sum(e[0] for e in each), flops=sum(e[1] for e in each))
    if kind in ("newton", "errors"):
        nr, nx, ny = case.get("nret", 1), case["nx"], case["ny"]
        b = nr * (4.0 * nx * ny + 8.0 * nx * nx + 16.0 * ny + 12.0 * nx)
        f = nr * (2.0 * nx * nx * ny + nx ** 3 / 3.0 + 4.0 * nx * ny)
        if kind == "errors":
            b += 8.0 * nx * ny + 8.0 * nx * nx + 12.0 * nx * nx
            f += 6.0 * nx * nx * ny + 4.0 * nx ** 3
        return dict(bytes=b, flops=f)
    if kind == "conv":
        n, w, c = case["nser"], case["nwave"], case["nconv"]
        return dict(bytes=4.0 * (n * w + w + c + n * c), flops=n * (20.0 * w + 20.0 * 25 * c))
    # retrievals: about five forward calls and Newton steps each
    j = dict(case, kind="spectrum", angle=0.0)
    b, f = _forward_work(_spectrum_job(j, 1), case["ng"])
    nx, ny = case["nlayer"] + case["ngas"], case["nwave"]
    return dict(bytes=case["nret"] * 5 * b, flops=case["nret"] * 5 * (f + 2.0 * nx * nx * ny + nx ** 3 / 3.0))


# ------------------------------------------------------------ 64-bit values
def _overlap64(k, cols, k2, dk2, a2, delg):
    """Random overlap of the distribution k [W, L, g] with k2 * a2 (the gas is
    added): sorted sums rebinned to the g-ordinates; cols [c, W, L, g] are the
    gradient columns, the last of them d/dT; the added gas's column goes in
    before it."""
    ng = len(delg)
    W, L = k.shape[:2]
    n = ng * ng
    row = lambda x: x[..., :, None].expand(*x.shape, ng).reshape(*x.shape[:-1], n)
    col = lambda x: x[..., None, :].expand(*x.shape[:-1], ng, ng).reshape(*x.shape[:-1], n)
    key, order = torch.sort(row(k) + col(k2 * a2), dim=-1, stable=True)
    w = (delg[:, None] * delg[None, :]).reshape(n)[order]
    G = torch.cumsum(w, -1)
    g = torch.cumsum(delg, 0)
    gb = g[:-1].expand(W, L, ng - 1).contiguous()
    p = torch.searchsorted(G, gb).clamp(max=n - 1)
    G0 = torch.where(p > 0, torch.gather(G, -1, (p - 1).clamp(min=0)), torch.zeros_like(gb))
    share = gb - G0                                        # the part of the split element below the boundary
    edge = torch.cat([torch.zeros_like(G[..., :1]), gb, G[..., -1:]], -1)
    width = edge[..., 1:] - edge[..., :-1]

    def rebin(v):
        c = torch.cumsum(w * v, -1)
        at = torch.where(p > 0, torch.gather(c, -1, (p - 1).clamp(min=0)), torch.zeros_like(gb)) + share * torch.gather(v, -1, p)
        i = torch.cat([torch.zeros_like(c[..., :1]), at, c[..., -1:]], -1)
        return (i[..., 1:] - i[..., :-1]) / width

    vs = [row(c) for c in cols[:-1]] + [col(k2), row(cols[-1]) + col(dk2 * a2)]
    return rebin(key), [rebin(torch.gather(v, -1, order)) for v in vs]


def _layer_grid(kt, job):
    """Position of the layers in the (ln p, T) grid of the tables."""
    f = lambda x: torch.tensor(np.asarray(x, np.float64), device=DEV)
    lnp, tk = f(kt.lnp), f(kt.tk)

    def place(grid, x):
        x = torch.minimum(torch.maximum(x, grid[0]), grid[-1])
        i = (torch.searchsorted(grid, x, right=True) - 1).clamp(0, len(grid) - 2)
        return i, (x - grid[i]) / (grid[i + 1] - grid[i]), 1.0 / (grid[i + 1] - grid[i])

    ip, v, _ = place(lnp, torch.log(f(job.press[:job.nlayer])))
    it, u, dudt = place(tk, f(job.temp[:job.nlayer]))
    return ip, it, u, v, dudt


def _forward64(kt, cia, job, per_position=False):
    """Radiance, Jacobian and d/dTsurf of a nadir-type job (IMOD 3, the job's
    one path, coincident wavenumbers), in 64 bits."""
    f = lambda x: torch.tensor(np.asarray(x, np.float64), device=DEV)
    L, na, ngas = job.nlayer, job.ngas - 2, job.ngas
    ng, nparam = kt.ng, job.nparam
    delg = f(kt.delg)
    ip, it, u, v, dudt = _layer_grid(kt, job)
    amount, pp, press, temp = f(job.amount[:L]), f(job.pp[:L]), f(job.press[:L]), f(job.temp[:L])
    utotl = amount.sum(1) * 1e-20
    # CIA (H2-H2 and H2-He, the pairs the table holds)
    big = pp.argmax(1)
    pick = lambda m: m.gather(1, big[:, None])[:, 0]
    height = f(job.delh[:L]) * 1e5
    tau_cia = height * ((pick(amount) * press / pick(pp) / height) / float(np.float32(2.68675e19))) ** 2
    qh2, qhe = pp[:, 0] / press, pp[:, 1] / press
    kc = torch.tensor(cia.kcia.reshape((9, 25, -1), order="F").astype(np.float64), device=DEV)
    tg = f(cia.temps.astype(np.float32))
    ct = (torch.searchsorted(tg, temp, right=True) - 1).clamp(0, 23)
    cu, cdu = (temp - tg[ct]) / (tg[ct + 1] - tg[ct]), 1.0 / (tg[ct + 1] - tg[ct])
    layinc = torch.tensor(job.layinc[:L, 0].astype(np.int64) - 1, device=DEV)
    scale, emt = f(job.scale[:L, 0]), f(job.emtemp[:L, 0])
    bins = np.rint((job.vwave.astype(np.float64) - float(kt.vmin[0])) / float(kt.delv[0])).astype(np.int64)
    tabs = [torch.from_numpy(kt.table(int(job.ktab[2 + a]))[bins]).to(DEV) for a in range(na)]
    x0 = 1.0
    if job.iform == 3:
        pi = float(np.float32(3.1415927))
        x0 = pi * 4.0 * pi * (float(np.float32(job.radius1)) * 1e5) ** 2 * float(np.float32(1e-18))
    dam, dte = f(job.dam[:L]), f(job.dte[:L])
    xmap = f(job.xmap)
    rad, gts, jac, dqs = [], [], [], []
    chunk = max(1, int((120 if DEV == "cuda" else 12) * 1000 / L))
    for w0 in range(0, job.nwave, chunk):
        vw = f(job.vwave[w0:w0 + chunk])
        W = len(vw)
        k, cols = None, None
        for a in range(na):
            t = tabs[a][w0:w0 + chunk].double()
            corner = lambda dp, dt: torch.log(t[:, ip + dp, it + dt, :])
            y1, y2, y3, y4 = corner(0, 0), corner(1, 0), corner(1, 1), corner(0, 1)
            V, U = v[None, :, None], u[None, :, None]
            k2 = torch.exp((1 - V) * (1 - U) * y1 + V * (1 - U) * y2 + V * U * y3 + (1 - V) * U * y4)
            dk2 = k2 * ((1 - V) * (y4 - y1) + V * (y3 - y2)) * dudt[None, :, None]
            a2 = (amount[:, 2 + a] * 1e-20)[None, :, None]
            if k is None:
                k, cols = k2 * a2, [k2, dk2 * a2]
            else:
                k, cols = _overlap64(k, cols, k2, dk2, a2, delg)
        # continuum
        cv = torch.floor(vw / cia.dnu).long().clamp(0, kc.shape[2] - 2)
        ft = (vw / cia.dnu - cv)[:, None]
        at = lambda q, dt, dv: kc[q, (ct + dt)[None, :], (cv + dv)[:, None]]
        al, da = [], []
        for q in (0, 1):
            a11, a12, a22, a21 = at(q, 0, 0), at(q, 0, 1), at(q, 1, 1), at(q, 1, 0)
            al.append((1 - ft) * (1 - cu) * a11 + ft * (1 - cu) * a12 + ft * cu * a22 + (1 - ft) * cu * a21)
            da.append(((1 - ft) * (a21 - a11) + ft * (a22 - a12)) * cdu)
        dtau = torch.zeros(nparam, W, L, ng, dtype=torch.float64, device=DEV)
        tau = (qh2 * qh2 * al[0] + qh2 * qhe * al[1]) * tau_cia
        dtau[0] += ((2 * qh2 * al[0] + qhe * al[1]) * tau_cia / (utotl * 1e20))[..., None]
        dtau[1] += (qh2 * al[1] * tau_cia / (utotl * 1e20))[..., None]
        dtau[ngas] += ((qh2 * qh2 * da[0] + qh2 * qhe * da[1]) * tau_cia)[..., None]
        for d in range(job.ncont):
            xs = f(job.xsec_ext[d, w0:w0 + chunk])[:, None]
            tau = tau + xs * f(job.cont[d, :L])[None, :]
            dtau[ngas + 1 + d] += xs[..., None]
        tau = tau[..., None] + k
        for a in range(na):
            dtau[2 + a] += cols[a] * 1e-20
        dtau[ngas] += cols[-1]
        # the path: emission, transmission and their derivatives
        ts = tau[:, layinc] * scale[None, :, None]
        tr = torch.exp(-torch.cumsum(ts, 1))
        tr0 = torch.cat([torch.ones_like(tr[:, :1]), tr[:, :-1]], 1)
        td = tr0 * -torch.expm1(-ts)
        c1, c2 = float(np.float32(1.1911e-12)), float(np.float32(1.439))
        x = c2 * vw[:, None] / emt[None, :]
        B = c1 * vw[:, None] ** 3 / torch.expm1(x)
        dB = B * (x / emt[None, :]) * torch.exp(x) / torch.expm1(x)
        ground = B[:, -1][:, None] * tr[:, -1]
        R = (td * B[..., None]).sum(1) + ground
        below = torch.flip(torch.cumsum(torch.flip(td * B[..., None], (1,)), 1), (1,)) - td * B[..., None]
        drdt = B[..., None] * tr - below - ground[:, None]
        rad.append(x0 * (R @ delg))
        gts.append(x0 * ((tr[:, -1] * dB[:, -1][:, None]) @ delg))
        dq = torch.einsum("wjg,pwjg,g->pwj", drdt, dtau[:, :, layinc] * scale[None, None, :, None], delg)
        dq[ngas] += torch.einsum("wjg,wj,g->wj", td, dB, delg)
        dq = dq * x0
        if per_position:
            dqs.append(dq)
            continue
        out = torch.zeros(job.nv, W, dtype=torch.float64, device=DEV)
        for p in range(nparam):
            if bool((job.xmap[:, p] != 0).any()):
                M = f(job.dco[:L]) if p > ngas else dte if p == ngas else dam
                out += torch.einsum("vr,wr->vw", xmap[:, p], dq[p] @ M[layinc])
        jac.append(out)
    rad, gts = torch.cat(rad).cpu().numpy(), torch.cat(gts).cpu().numpy()
    if per_position:
        return rad, gts, torch.cat(dqs, 1).cpu().numpy()
    jac = torch.cat(jac, 1).cpu().numpy()
    if job.conv is not None:
        c = _convolve64(job.vwave, np.concatenate([rad[None], gts[None], jac]), job.fwhm, job.conv.vconv)
        rad, gts, jac = c[0], c[1], c[2:]
    return rad, jac.ravel(), gts


def _convolve64(v, y, fwhm, vconv):
    """Natural cubic spline through the points, 20 points across each channel's square bin, trapezoid."""
    v, y, vc = v.astype(np.float64), np.atleast_2d(y).astype(np.float64), vconv.astype(np.float64)
    fwhm = float(np.float32(fwhm))
    n, h = len(v), np.diff(v)
    A = np.diag(np.r_[1.0, 2 * (h[:-1] + h[1:]), 1.0])
    A[np.arange(1, n - 1), np.arange(0, n - 2)] = h[:-1]
    A[np.arange(1, n - 1), np.arange(2, n)] = h[1:]
    rhs = np.zeros((n, y.shape[0]))
    s = np.diff(y, axis=1) / h
    rhs[1:-1] = 6.0 * (s[:, 1:] - s[:, :-1]).T
    y2 = np.linalg.solve(A, rhs).T
    x = vc[:, None] - fwhm / 2 + np.arange(20)[None, :] * (fwhm / 19)
    i = np.clip(np.searchsorted(v, x, side="right") - 1, 0, n - 2)
    a = (v[i + 1] - x) / h[i]
    b = (x - v[i]) / h[i]
    f = a * y[:, i] + b * y[:, i + 1] + ((a ** 3 - a) * y2[:, i] + (b ** 3 - b) * y2[:, i + 1]) * h[i] ** 2 / 6.0
    return (f[..., 1:] + f[..., :-1]).sum(-1) * (fwhm / 38) / fwhm


def exact(case, seed):
    kind = case["kind"]
    if kind == "wave":
        rad, gts, dq = _forward64(_tables_for(case), _cia(), _spectrum_job(case, seed), per_position=True)
        dq[:2] = 0.0                        # H2 and He are not among the asked parameters
        return rad, gts, np.transpose(dq, (1, 2, 0))
    if kind == "spectrum":
        return _forward64(_tables_for(case), _cia(), _spectrum_job(case, seed))
    if kind in ("batch", "resident"):
        return [_forward64(_tables_for(case), _cia(), j) for j in _batch_jobs(case, seed)]
    if kind in ("newton", "errors"):
        d = _oe_inputs(case.get("nret", 1), case["nx"], case["ny"], seed)
        f = lambda x: np.asarray(x, np.float64)
        xs, phis, chis = [], [], []
        for r in range(case.get("nret", 1)):
            kk, sei, sai = f(d["kk"][r]), d["sei"][r], d["sai"][r]
            C = (kk * sei) @ kk.T + sai
            dy, dx = f(d["y"][r]) - f(d["yn"][r]), f(d["xn"][r]) - f(d["xa"][r])
            xs.append(f(d["xa"][r]) + np.linalg.solve(C, kk @ (sei * (dy + kk.T @ dx))))
            chis.append((sei * dy * dy).sum())
            phis.append(chis[-1] + dx @ sai @ dx)
        if kind == "newton":
            return np.stack(xs), None, np.array(phis), np.array(chis)
        dd = np.linalg.solve(C, kk * sei)
        aa = dd @ kk.T
        sm = (dd / sei) @ dd.T
        e = aa - np.eye(case["nx"])
        sn = e @ f(d["sa"]) @ e.T
        return xs[0], None, dd, aa, sn + sm, sn, sm
    if kind == "conv":
        v, y, ch = _conv_inputs(case, seed)
        return _convolve64(v, y, case["fwhm"], ch.vconv)
    return None                             # a whole iteration: its steps are the cases above
