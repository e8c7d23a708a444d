"""The work a simulation has this library do, as timed cases.

One run of the code is a loop over output times: an interval of leapfrog
steps, then the outputs (defect counts and fits, GW spectrum, field spectrum),
for one lattice or for an ensemble of them, and now and then a gradient run.
Each case below is one such call or short sequence of calls through the
package's public entry points, over the lattice sizes, precisions and GW
methods the tests, the benchmark and its configurations use.

The fields are seeded band-limited Gaussian fields of unit mean square (what
ic_gaussian_flat draws), made here on the GPU with torch, and for the output
calls evolved by the library to the age at which such a call is made.

Kinds:
  interval   upload phi, phi' from the host's arrays, `steps` leapfrog steps
             of phi and six u_ij, download phi and phi' (and u_ij, u'_ij on
             small lattices): the drop-in use, where the host program holds
             data1 / data2 and the library steps them between output times
  green      steps with the Green's-function GW integration, then its spectrum
  gw         the two GW spectra (linear and log bins) of the u_ij state
  defects    cell classification and plaquette winding, the counts
  fits       id_defects with every string and wall fit, and the fitted lists
  spectrum   classification, masked field spectrum with deconvolution, rho
  adjoint    gradient of the band-integrated GW energy
  ensemble   a graph-replayed interval of several lattices of uneven sizes in
             one batch, and the mean GW spectrum over the members
"""
import ctypes
import math

import numpy as np
import torch

import axion_grav_gb300 as ag

PRECISION = {"fp64": ag.PREC_FP64_PLAIN, "fused": ag.PREC_FP64_FUSED, "fp32": ag.PREC_FP32_MIXED}
EPS = 0.25  # eps_dtau of the workloads
T0 = 2.0  # conformal time the steps start at
TAU_CR = 1e20  # tau_cr in reduced-Planck units: GW powers of order one
PI = 3.14159265359  # the library's pi (potential.f90:8) in bins and wave numbers
UIJ_DOWNLOAD = 128  # largest lattice whose u_ij an interval returns


def listed():
    return [
        # the smallest lattice a test or a quick scan steps: launches and latency
        dict(name="interval_32_fp32", kind="interval", n=32, precision="fp32", steps=20),
        # a lattice size that is no multiple of 32 (box sizes chosen by physics)
        dict(name="interval_100_fp32", kind="interval", n=100, precision="fp32", steps=20),
        # the drop-in at the reference's precision, the 128^3 plain-method workload
        dict(name="interval_128_fp64", kind="interval", n=128, precision="fp64", steps=20),
        # the headline lattice, 20 steps between output times
        dict(name="interval_512_fp32", kind="interval", n=512, precision="fp32", steps=20),
        # Green's-function GW mode, the reference's own GW method
        dict(name="green_512_fp32", kind="green", n=512, precision="fp32", steps=4),
        dict(name="green_256_fp64", kind="green", n=256, precision="fp64", steps=4),
        # the outputs of one output time
        dict(name="gw_512_fp32", kind="gw", n=512, precision="fp32", steps=8),
        dict(name="defects_512_fp32", kind="defects", n=512, precision="fp32", steps=40),
        dict(name="fits_128_fp32", kind="fits", n=128, precision="fp32", steps=24),
        dict(name="spectrum_256_fp32", kind="spectrum", n=256, precision="fp32", steps=24, degrade=0),
        # gradient run (forward with checkpoints, reverse sweep)
        dict(name="adjoint_128_fp32", kind="adjoint", n=128, precision="fp32", steps=48, stride=16),
        # many realisations of uneven sizes in one batch
        dict(name="ensemble_fp32", kind="ensemble", n=160, precision="fp32", steps=10, members=8),
    ]


def _even(rng, lo, hi):
    """An even lattice size, log-uniform in [lo, hi]: half of them multiples of 32."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if rng.random() < 0.5 and n >= 24:
        return min(hi, max(32, 32 * round(n / 32)))
    return max(lo, min(hi, 2 * round(n / 2)))


def draw(rng):
    kind = rng.choice(["interval", "interval", "green", "gw", "defects", "fits", "spectrum", "adjoint", "ensemble"])
    prec = rng.choice(["fp32", "fp64", "fused", "fp32"])
    if kind == "interval":
        return dict(kind=kind, n=_even(rng, 16, 416 if prec == "fp32" else 192), precision=prec,
                    steps=rng.randint(1, 24 if prec == "fp32" else 16))
    if kind == "green":
        return dict(kind=kind, n=_even(rng, 24, 384 if prec == "fp32" else 208), precision=prec, steps=rng.randint(1, 4))
    if kind == "gw":
        return dict(kind=kind, n=_even(rng, 24, 416 if prec == "fp32" else 288), precision=prec, steps=rng.randint(4, 8))
    if kind == "defects":
        return dict(kind=kind, n=_even(rng, 24, 448), precision=prec, steps=rng.randint(8, 40))
    if kind == "fits":
        return dict(kind=kind, n=_even(rng, 24, 112), precision=prec, steps=rng.randint(16, 24))
    if kind == "spectrum":
        deg = rng.choice([0, 0, 1])
        n = _even(rng, 48, 224)
        return dict(kind=kind, n=n - n % (2 << deg), precision=prec, steps=rng.randint(8, 24), degrade=deg)
    if kind == "adjoint":
        steps = rng.randint(8, 32)
        return dict(kind=kind, n=_even(rng, 32, 112), precision="fp32" if prec == "fused" else prec, steps=steps,
                    stride=rng.randint(4, steps))
    return dict(kind=kind, n=32 * rng.randint(2, 5), precision="fused" if prec == "fp64" else prec,
                steps=rng.randint(4, 12), members=rng.randint(3, 10))


# ---- fields ---------------------------------------------------------------


def _field(n, seed, frac=0.125):
    """Complex Gaussian field, modes up to `frac` of 2 pi / dx, <|phi|^2> = 1."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = torch.fft.fftn(torch.view_as_complex(torch.randn(n, n, n, 2, dtype=torch.float64, device="cuda", generator=g)))
    k = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    f *= k2 <= frac * frac + 1e-12
    del k2
    f = torch.fft.ifftn(f)
    return f / torch.sqrt(torch.mean(torch.view_as_real(f).square()) * 2)


def _array(shape, dtype=torch.complex128):
    """An array of the host program, in pinned memory."""
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _host(phi):
    """The host program's array holding the field."""
    return torch.empty(phi.shape, dtype=phi.dtype, pin_memory=True).copy_(phi).numpy()


def _sizes(case):
    """Member sizes of an ensemble: the largest, and smaller multiples of 32."""
    return [max(32, case["n"] - 32 * (i % 4)) for i in range(case["members"])]


def _params(case, n=None, seed=1):
    n = n or case["n"]
    kind = case["kind"]
    gw = {"green": ag.GW_GREEN, "defects": ag.GW_NONE, "fits": ag.GW_NONE, "spectrum": ag.GW_NONE}.get(kind, ag.GW_UIJ)
    kw = dict(ngrid=n, precision=PRECISION[case["precision"]], gw_mode=gw, compat=ag.COMPAT_INTENDED, tau_cr=TAU_CR,
              seed=seed, degrade_spec=case.get("degrade", 0), flags=7)
    if kind in ("adjoint",):  # the quartic model of the gradient workload
        kw.update(potential=ag.POT_QUARTIC, dspa=1.0, sigma_cr=0.005, vev=1.0, **{"lambda": 1.0})
    elif kind == "ensemble":
        kw.update(potential=ag.POT_REFERENCE, dspa=0.5, sigma_cr=1.0, kappa=0.1)
    else:
        kw.update(potential=ag.POT_REFERENCE, dspa=32.0 / n, sigma_cr=1.0, kappa=0.1)
    return ag.default_params(**kw)


def _dt(case, p):
    if case["kind"] == "adjoint":
        return 0.2
    if case["kind"] == "ensemble":
        return 0.05
    # get_dtau (evolve.f90:10-24) over the run [2, 32]
    n = p.ngrid
    omega = math.hypot(2 * PI / p.dspa / n * n, 2.449489742783178 * 32.0 * p.sigma_cr)
    return 30.0 / max(1, math.ceil(30.0 / (EPS / omega)))


def _new_lattice(case, seed):
    p = _params(case, seed=seed)
    lat = ag.Lattice(p)
    phi = _host(_field(case["n"], seed))
    lat.upload(phi, np.zeros_like(phi))
    return lat, p


def _dp(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    st = dict(case=case)
    if kind == "ensemble":
        sizes = _sizes(case)
        ens = ag.Ensemble([_params(case, m, seed + i) for i, m in enumerate(sizes)])
        for i, m in enumerate(sizes):
            phi = _host(_field(m, seed * 64 + i))
            ens.member(i).upload(phi, np.zeros_like(phi))
        st.update(ens=ens, p=_params(case))
        return st
    if kind == "interval":
        p = _params(case, seed=seed)
        st.update(lat=ag.Lattice(p), phi=_host(_field(n, seed)), phid=_host(0.1 * _field(n, seed + 7919)))
        # the host program's own result arrays
        st.update(out=_array((2, n, n, n)))
        if n <= UIJ_DOWNLOAD:
            st.update(out_u=_array((2, 6, n, n, n), torch.float64))
    elif kind == "adjoint":
        p = _params(case, seed=seed)
        st.update(lat=ag.Lattice(p), phi=_host(_field(n, seed)), zero=_array(6 * n ** 3, torch.float64))
    else:
        lat, p = _new_lattice(case, seed)
        if kind != "green":
            lat.leapfrog(T0, _dt(case, p), case["steps"])
        st.update(lat=lat)
        if kind == "fits":  # room for the fitted cells
            st.update(strings=_array((n ** 3 // 8, 13), torch.float64), walls=_array((n ** 3 // 2, 10), torch.float64))
    st.update(p=p, dt=_dt(case, p))
    return st


def _spectrum_of(case, wave_free):
    """Spectra of FP32-mixed states carry 32-bit fields' digits: handed on as such."""
    t = np.float32 if case["precision"] == "fp32" else np.float64
    return [np.asarray(v, t) for v in wave_free]


def run(st):
    case = st["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        st["ens"].leapfrog(T0, _dt(case, st["p"]), steps)
        w, m, s, d = st["ens"].grav_spec_mean(T0 + steps * _dt(case, st["p"]))
        return dict(power=_spectrum_of(case, [m, s]), modes=d)
    lat, p, dt = st["lat"], st["p"], st["dt"]
    tau = T0 + steps * dt
    if kind == "interval":
        n = case["n"]
        lat.upload(st["phi"], st["phid"])
        lat.leapfrog(T0, dt, steps)
        out = st["out"]
        lat._check(lat.lib.axg_download(lat.handle, _dp(out[0]), _dp(out[1]), n * n, 0))
        if "out_u" not in st:
            return dict(phi=out[0], phid=out[1])
        u = st["out_u"]
        lat._check(lat.lib.axg_download_uij(lat.handle, _dp(u[0]), _dp(u[1])))
        return dict(phi=out[0], phid=out[1], u=u[0], ud=u[1])
    if kind == "green":
        lat.leapfrog(T0, dt, steps)
        w, pw, nu, de = lat.grav_spec_estimation(tau)
        return dict(power=_spectrum_of(case, [pw, nu]), modes=de)
    if kind == "gw":
        w, pw, nu, de = lat.grav_spec_estimation(tau)
        e, lpw, lnu, lde = lat.grav_spec_log(tau)
        return dict(power=_spectrum_of(case, [pw, nu, lpw, lnu]), modes=[de, lde])
    if kind == "defects":
        return dict(counts=lat.classify_cells(7), winding=lat.string_winding())
    if kind == "fits":
        sl, wa, sv, c = lat.id_defects(1, tau)
        s, w = st["strings"], st["walls"]
        lat._check(lat.lib.axg_download_defect_lists(lat.handle, _dp(s), len(s), _dp(w), len(w)))
        return dict(length=sl, area=wa, velocity=sv, counts=c, strings=s, walls=w)
    if kind == "spectrum":
        c = lat.classify_cells(7)
        w, pw, cv, ct = lat.spectrum_estimation(tau)
        return dict(counts=c, power=pw, conv=cv, modes=ct, rho=lat.compute_crho())
    zero = st["zero"]  # phi' = 0, u_ij = u'_ij = 0
    lat.upload(st["phi"], zero[: 2 * case["n"] ** 3].view(np.complex128))
    lat.upload_uij(zero, zero)
    J, dl, g0, g1, _, _ = lat.adjoint_gw_band(1.0, dt, steps, case["stride"], 0.125, 0.5)
    return dict(J=J, dlambda=dl, grad_phi=g0, grad_phid=g1)


def work(case):
    """Least traffic of a pass: state in and out once per step, each spectrum
    from its fields once, each defect pass phi in and its result out once."""
    n, kind, steps = case["n"], case["kind"], case["steps"]
    n3, f32 = float(n) ** 3, case["precision"] == "fp32"
    step = 192.0 if f32 else (384.0 if case["precision"] == "fp64" else 256.0)
    step_phi = 48.0 if f32 else (96.0 if case["precision"] == "fp64" else 64.0)
    ops = 150.0  # operations of one site-update (phi and six u_ij)
    fft = 2.5 * math.log2(n3)  # operations per real site of a real transform
    if kind == "ensemble":
        sites = float(sum(m ** 3 for m in _sizes(case)))
        return dict(bytes=sites * (step * steps + (72.0 if f32 else 96.0)), flops=sites * (ops * steps + 12 * fft))
    if kind == "interval":
        extra = 96.0 if n <= UIJ_DOWNLOAD else 0.0
        return dict(bytes=n3 * (step * steps + 64.0 + extra), flops=n3 * ops * steps)
    if kind == "green":  # phi step; phi and the accumulators of half the modes in and out
        acc = 64.0 + (8.0 if f32 else 16.0)
        return dict(bytes=n3 * (step_phi + acc) * steps, flops=n3 * steps * (45.0 + 6 * fft + 60.0))
    if kind == "gw":
        return dict(bytes=2 * n3 * (72.0 if f32 else 96.0), flops=2 * n3 * (12 * fft + 60.0))
    if kind == "defects":
        return dict(bytes=n3 * (2 * (8.0 if f32 else 16.0) + 1.0), flops=n3 * 120.0)
    if kind == "fits":
        # a few per cent of the cells, ~700 evaluations of the fit function each
        return dict(bytes=n3 * 17.0, flops=n3 * 0.06 * 700 * 400)
    if kind == "spectrum":
        m3 = n3 / 8 ** case["degrade"]
        return dict(bytes=n3 * (16.0 if f32 else 32.0) + m3 * 8, flops=m3 * 3 * 2.5 * math.log2(m3))
    return dict(bytes=n3 * steps * (192.0 + 240.0 if f32 else 384.0 + 480.0), flops=n3 * steps * (ops + 250.0))


# ---- the same outputs in 64 bits from plain torch ---------------------------


def _coef(p, t, dt):
    """Kick coefficients (evolve.f90:291-305) and dV/dphi* = (A |phi|^2 + B) phi + C."""
    h = dt / t
    f = [(1 - h) / (1 + h), dt / p.dspa ** 2 / (1 + h), -dt * t * t * p.sigma_cr ** 2 / (1 + h),
         dt * p.sigma_cr ** 2 / (1 + h)]
    if p.potential == ag.POT_QUARTIC:
        return f, p.lambda_ / 2, -p.lambda_ * p.vev ** 2 / 2, 0.0
    s = 2.449489742783178
    th, k2 = s / t, p.kappa * p.kappa
    m = 6.26 * (p.kappa / th) ** 6.68 if th > p.kappa * 6.26 ** (1 / 6.68) else 1.0
    return f, 2.0, (th * th - s * s) / 3, -m * k2 * k2 / 2


def _lap(a):
    r = -6 * a
    for d in (-1, -2, -3):
        r = r + torch.roll(a, 1, d) + torch.roll(a, -1, d)
    return r


def _sources(phi, dx):
    g = [(torch.roll(phi, -1, d) - torch.roll(phi, 1, d)) / (2 * dx) for d in (-1, -2, -3)]
    return [2 * (g[i].real * g[j].real + g[i].imag * g[j].imag) for i in range(3) for j in range(i + 1)]


def _evolve(p, phi, phid, u, ud, t, dt, steps, each=None, lam=None):
    """Drift-kick-drift of phi (and of u, ud, [6, n, n, n], unless None)."""
    phi = phi + dt / 2 * phid
    u = u if u is None else u + dt / 2 * ud
    t = t + dt / 2
    for it in range(steps):
        f, A, B, C = _coef(p, t, dt)
        if lam is not None:
            A, B = lam / 2, -lam * p.vev ** 2 / 2
        if each is not None:
            each(phi, t)
        h = dt / 2 if it == steps - 1 else dt
        ddv = (A * (phi.real ** 2 + phi.imag ** 2) + B) * phi + C
        if u is not None:
            S = _sources(phi, p.dspa)
            ud = torch.stack([f[0] * ud[c] + f[1] * _lap(u[c]) + f[3] * S[c] for c in range(6)])
            u = u + h * ud
        phid = f[0] * phid + f[1] * _lap(phi) + f[2] * ddv
        phi = phi + h * phid
        t = t + h
    return phi, phid, u, ud


def _kgrid(n, half):
    j = torch.arange(n, device="cuda", dtype=torch.float64)
    k = torch.remainder(j + n // 2, n) - n // 2
    kx = k[: n // 2 + 1] if half else k
    return kx[None, None, :], k[None, :, None], k[:, None, None]


def _bins(k2, dwav, dx, nb, log):
    """Bin of each |k|^2 (nb: outside): linear (grav_waves.f90:279) or log on [dwav, pi / dx]."""
    q = torch.sqrt(k2) * dwav
    if log:
        qmax = PI / dx
        e = [dwav * math.pow(qmax / dwav, k / nb) for k in range(nb + 1)]
        b = torch.bucketize(q, torch.tensor(e, dtype=torch.float64, device="cuda"), right=True) - 1
        b = torch.where(q == e[nb], nb - 1, b)
        bad = (q < e[0]) | (q > e[nb])
    else:
        b = torch.floor(q / (PI / dx / nb) + 1.0).long() - 1
        bad = b >= nb
    return torch.where(bad | (q <= 0), nb, b)


def _sum_bins(b, v, nb):
    return torch.bincount(b.reshape(-1), weights=v.reshape(-1), minlength=nb + 1)[:nb].cpu().numpy()


def _tt(U, kk, kq):
    """|TT projection|^2 per k of a symmetric tensor spectrum (11, 21, 22, 31, 32, 33)."""
    h = [c / kq for c in kk]
    idx = [[0, 1, 3], [1, 2, 4], [3, 4, 5]]
    s, tot, lin = 0, 0, 0
    for i in range(3):
        v = sum(U[idx[i][j]] * h[j] for j in range(3))
        s = s + v * h[i]
        lin = lin + v.real ** 2 + v.imag ** 2
        for j in range(3):
            w = U[idx[i][j]]
            tot = tot + w.real ** 2 + w.imag ** 2
    d = U[0] + U[2] + U[5] - s
    return tot - 2 * lin + s.real ** 2 + s.imag ** 2 - 0.5 * (d.real ** 2 + d.imag ** 2)


def _gw_energy(p, u, ud, tau):
    """(weights per half-spectrum k, |k|^2, energy |W'_TT|^2 + k^2 |W_TT|^2)."""
    n = p.ngrid
    kk = _kgrid(n, True)
    k2 = kk[0] ** 2 + kk[1] ** 2 + kk[2] ** 2
    kq = torch.sqrt(k2).clamp(min=0.5)
    dwav, dv = 2 * PI / p.dspa / n, p.dspa ** 3
    e = _tt([torch.fft.rfftn(u[c] + tau * ud[c]) for c in range(6)], kk, kq)
    e = e + k2 * dwav ** 2 * _tt([torch.fft.rfftn(tau * u[c]) for c in range(6)], kk, kq)
    wgt = torch.full((n // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    wgt[0] = wgt[-1] = 1.0
    return wgt[None, None, :].expand(k2.shape), k2, e * (dv * dv)


def _gw_spectrum(p, wgt, k2, e, log):
    n, nb = p.ngrid, p.gw_log_bins if log else p.num_bin_grav
    dwav, qmax = 2 * PI / p.dspa / n, PI / p.dspa
    b = _bins(k2, dwav, p.dspa, nb, log)
    nu, de = _sum_bins(b, wgt * e, nb), _sum_bins(b, wgt, nb)
    if log:
        x = np.array([dwav * math.pow(qmax / dwav, k / nb) for k in range(nb + 1)])
        qc = np.sqrt(x[1:] * x[:-1])
    else:
        qc = (np.arange(nb) + 0.5) * (qmax / nb)
    fact = 1 / p.tau_cr ** 6 / (2.1332e-42 / 2.435e18) ** 2 / p.a_now ** 4 / 3 / (2 * PI) ** 2 * (dwav / 2 / PI) ** 3
    return np.where(de > 0, nu / np.maximum(de, 1) * qc ** 3 * fact, 0.0), nu, de


def _mask(phi):
    """Cells whose largest circular phase gap is below 7 pi / 4 (defects_3d.f90:309-349)."""
    ph = torch.angle(phi)
    c = [torch.roll(ph, (-dz, -dy, -dx), (0, 1, 2)) for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)]
    s = torch.sort(torch.stack(c, -1), -1).values
    t, g = s[..., 0] - s[..., 7] + 2 * PI, (s[..., 1:] - s[..., :-1]).amax(-1)
    return torch.where(g > t, g, torch.maximum(g, t)) < 7 * PI / 4


def _coupling(p, m, w2, cnt):
    """Mode-coupling matrix of the window (spectrum.f90:74-98, 117-171, 344-444) from
    the |k|^2 histograms of |W|^2 and of the modes."""
    nb, dx = p.num_bin, p.dspa * 2 ** p.degrade_spec
    dq, dwav = PI / dx / nb, 2 * PI / dx / m
    q = torch.sqrt(torch.arange(len(w2), dtype=torch.float64, device="cuda")) * dwav
    ip = torch.arange(1, 201, dtype=torch.float64, device="cuda") - 0.5
    mat = torch.zeros(nb, nb, dtype=torch.float64, device="cuda")
    wav = [k * dq for k in range(nb + 1)]
    for i in range(nb):
        li, si = wav[i + 1], wav[i]
        for j in range(i + 1):
            lj, sj = wav[j + 1], wav[j]
            q0 = max(0.0, max(si, sj) - min(li, lj))
            d = (li + lj - q0) / 500
            x = (q0 + d * torch.arange(501, dtype=torch.float64, device="cuda"))[:, None]
            hi = torch.clamp(x + li, max=lj)
            lo = torch.maximum(torch.maximum(x - li, si - x), torch.full_like(x, sj))
            dp = (hi - lo) / 200
            pp = dp * ip + lo
            xs = torch.where(x == 0, torch.ones_like(x), x)
            up = torch.clamp((li * li - pp * pp - x * x) / 2 / pp / xs, max=1.0)
            dn = torch.clamp((si * si - pp * pp - x * x) / 2 / pp / xs, min=-1.0)
            up, dn = torch.where(x == 0, 1.0, up), torch.where(x == 0, -1.0, dn)
            tab = torch.where(dp[:, 0] > 0, (pp * pp * dp * (up - dn)).sum(1), 0.0) * 2 * PI
            r = (q - q0) / d
            fl = torch.floor(r)
            ok = (fl >= 0) & (fl < 500)
            k = torch.where(ok, fl, 0.0).long()
            fr = r - fl
            v = torch.where(ok, (1 - fr) * tab[k] + fr * tab[k + 1], 0.0)
            mat[i, j] = mat[j, i] = (w2 * v).sum() / (cnt * v).sum()
    return mat * (dwav / 2 / PI) ** 6


def _exact_spectrum(p, case, phi, phid, tau):
    n, deg, nb = case["n"], 1 << case["degrade"], p.num_bin
    m, dx = n // deg, p.dspa * deg
    dwav, dv = 2 * PI / dx / m, dx ** 3

    def coarse(a):
        return a.reshape(m, deg, m, deg, m, deg).sum((1, 3, 5))

    masked = coarse(_mask(phi).to(torch.float64)) > 0
    win = torch.where(masked, 0.0, dv)
    f = torch.where(masked, 0.0, coarse(phid) / deg ** 3)
    kk = _kgrid(m, False)
    k2 = kk[0] ** 2 + kk[1] ** 2 + kk[2] ** 2
    b = torch.floor(torch.sqrt(k2) * dwav / (PI / dx / nb) + 1.0).long() - 1
    b = torch.where(b >= nb, nb, b)
    F = torch.fft.fftn(f.conj()).abs().square() * (dv * dv * (dwav / 2 / PI) ** 3)
    ct = _sum_bins(b, torch.ones_like(k2), nb)
    cv = _sum_bins(b, F, nb) * tau * tau
    i2 = k2.long().reshape(-1)
    W = torch.fft.fftn(win).abs().square().reshape(-1)
    mat = _coupling(p, m, torch.bincount(i2, weights=W), torch.bincount(i2).to(torch.float64))
    inv = np.linalg.inv(mat.cpu().numpy()) / ct[:, None] / ct[None, :]
    pw = inv @ cv
    w = (np.arange(nb) + 0.5) * (PI / dx / nb)
    rho = float(np.sum(pw * w * w * (PI / dx / nb) / (2 * PI) / PI))
    return dict(counts=None, power=pw, conv=cv / ct, modes=ct, rho=rho)


def _exact_green(p, case, phi, dt):
    n, nb = case["n"], p.num_bin_grav
    kk = _kgrid(n, False)
    k2 = kk[0] ** 2 + kk[1] ** 2 + kk[2] ** 2
    kq = torch.sqrt(k2)
    dwav, dv = 2 * PI / p.dspa / n, p.dspa ** 3
    safe = kq.clamp(min=0.5)
    qx, qy, qz = (c / safe for c in kk)
    r = torch.sqrt(qx * qx + qy * qy).expand(k2.shape)
    rs = torch.where(r > 0, r, 1.0)
    c, s = torch.where(r > 0, qx / rs, 1.0), torch.where(r > 0, qy / rs, 0.0)
    pol = [torch.complex(qz * c, -s), torch.complex(qz * s, c), torch.complex(-r, torch.zeros_like(r))]
    del safe, rs, c, s, r
    acc = [torch.zeros(n, n, n, dtype=torch.complex128, device="cuda") for _ in range(4)]

    def kick(phi, t):
        xp = xm = 0
        S = _sources(phi, p.dspa)
        for idx, (i, j) in enumerate([(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2)]):
            F = torch.fft.fftn(S[idx]).conj() * (0.5 if i == j else 1.0)
            e = pol[i] * pol[j]
            xp = xp + e * F
            xm = xm + e.conj() * F
        dw = t * dt * dv * p.sigma_cr ** 2
        wc, ws = dw * torch.cos(kq * dwav * t), dw * torch.sin(kq * dwav * t)
        for a, (w, x) in enumerate([(wc, xp), (ws, xp), (wc, xm), (ws, xm)]):
            acc[a] += w * x

    _evolve(p, phi, torch.zeros_like(phi), None, None, T0, dt, case["steps"], kick)
    e = sum(a.real ** 2 + a.imag ** 2 for a in acc)
    pw, nu, de = _gw_spectrum(p, torch.ones_like(k2), k2, torch.where(k2 > 0, e, 0.0), False)
    return dict(power=[pw, nu], modes=de)


def _exact_adjoint(p, case, phi, dt):
    from torch.utils.checkpoint import checkpoint

    n = case["n"]
    x0 = torch.view_as_real(phi).clone().requires_grad_(True)
    x1 = torch.zeros_like(x0).requires_grad_(True)
    lam = torch.tensor(float(p.lambda_), dtype=torch.float64, device="cuda", requires_grad=True)

    def part(ph, pd, u, ud, lam, h0, t, h1):
        # one drift h0, the kick at t, and the drift h1 of the last step
        ph, u = torch.view_as_complex(ph.contiguous()), u + h0 * ud
        pd = torch.view_as_complex(pd.contiguous())
        ph = ph + h0 * pd
        f, _, _, C = _coef(p, t, dt)
        S = _sources(ph, p.dspa)
        ddv = (lam / 2 * (ph.real ** 2 + ph.imag ** 2) - lam * p.vev ** 2 / 2) * ph + C
        ud = torch.stack([f[0] * ud[c] + f[1] * _lap(u[c]) + f[3] * S[c] for c in range(6)])
        pd = f[0] * pd + f[1] * _lap(ph) + f[2] * ddv
        return torch.view_as_real(ph + h1 * pd), torch.view_as_real(pd), u + h1 * ud, ud

    ph, pd = x0, x1
    u = torch.zeros(6, n, n, n, dtype=torch.float64, device="cuda")
    ud = torch.zeros_like(u)
    t = 1.0
    for it in range(case["steps"]):
        h0 = dt / 2 if it == 0 else dt
        t = t + h0
        ph, pd, u, ud = checkpoint(part, ph, pd, u, ud, lam, h0, t, dt / 2 if it == case["steps"] - 1 else 0.0,
                                   use_reentrant=False)
    wgt, k2, e = _gw_energy(p, u, ud, 1.0 + dt * case["steps"])
    kk = torch.sqrt(k2) * (2 * PI / p.dspa / n)
    J = (0.5 * wgt * e * ((kk >= 0.125) & (kk <= 0.5) & (k2 > 0))).sum()
    J.backward()
    return dict(J=float(J), dlambda=float(lam.grad), grad_phi=torch.view_as_complex(x0.grad),
                grad_phid=torch.view_as_complex(x1.grad))


def exact(case, seed):
    kind, n, steps = case["kind"], case["n"], case["steps"]
    p = _params(case)
    dt = _dt(case, p)
    tau = T0 + steps * dt
    if kind in ("defects", "fits"):
        return None  # whole numbers; fits by a random search
    with torch.set_grad_enabled(kind == "adjoint"):
        if kind == "ensemble":
            pw = []
            for i, m in enumerate(_sizes(case)):
                q = _params(case, m)
                phi = _field(m, seed * 64 + i)
                z = torch.zeros(6, m, m, m, dtype=torch.float64, device="cuda")
                _, _, u, ud = _evolve(q, phi, torch.zeros_like(phi), z, z, T0, dt, steps)
                pw.append(_gw_spectrum(q, *_gw_energy(q, u, ud, tau), False))
            v, have = np.array([x[0] for x in pw]), np.array([x[2] > 0 for x in pw])
            k = np.maximum(have.sum(0), 1)
            mean = (v * have).sum(0) / k
            return dict(power=[mean, None], modes=sum(x[2] for x in pw))
        phi = _field(n, seed)
        if kind == "adjoint":
            return _exact_adjoint(p, case, phi, dt)
        if kind == "green":
            return _exact_green(p, case, phi, dt)
        uij = kind == "gw" or (kind == "interval" and n <= UIJ_DOWNLOAD)
        u = torch.zeros(6, n, n, n, dtype=torch.float64, device="cuda") if uij else None
        phid = 0.1 * _field(n, seed + 7919) if kind == "interval" else torch.zeros_like(phi)
        phi, phid, u, ud = _evolve(p, phi, phid, u, u, T0, dt, steps)
        if kind == "interval":
            return dict(phi=phi, phid=phid, u=u, ud=ud) if uij else dict(phi=phi, phid=phid)
        if kind == "gw":
            e = _gw_energy(p, u, ud, tau)
            a, b = _gw_spectrum(p, *e, False), _gw_spectrum(p, *e, True)
            return dict(power=[a[0], a[1], b[0], b[1]], modes=[a[2], b[2]])
        return _exact_spectrum(p, case, phi, phid, tau)
