"""The work that users of this solver have it do, as measurable cases.

Each case goes through a public entry point (`solve_case`, `solve_batch`,
`Plan`, `sos_reflectance`, `solve_batch_lut`, `solve_batch_ocean`) with inputs
drawn from its seed.  The sizes are those of the benchmark configurations, the
command-line defaults and the tests, and odd ones between them.

Outputs are the planes a program keeps of a solve, in FP32 (the precision the
radiation fields are computed in): reflectances and radiances as Stokes
vectors, transmittances, the spherical correction, the convergence flag,
gradients.  The iteration counters of the result record (`n_orders_used`,
`order_modes`, `orders_water`) describe how the sum was stopped, not what it
is, and are left out.

`exact` restates the plane-parallel solve over a black or rough surface in
FP64 with torch operations (and its gradients by autograd).
"""
import math

import numpy as np
import torch

BANDS = np.linspace(412.0, 865.0, 10)
WATER_BANDS = (412.0, 443.0, 490.0, 510.0, 555.0, 670.0, 765.0, 865.0)
DEPOL = 0.0279


def listed():
    return [
        # one pixel at the command line's defaults (24 streams, 40 layers, modes 0..2) over a
        # rough sea, no aerosol: an interactive call, a unit of a per-pixel loop
        dict(name="pixel", kind="single", streams=24, layers=40, modes=2, L=0, surface="rough", ipss=0),
        # one pixel with an aerosol at the reference's largest mode count, 400 layers
        dict(name="pixel_aerosol", kind="single", streams=32, layers=400, modes=32, L=120, surface="rough", ipss=0),
        # the same aerosol over every mode of its expansion (2L + 1), with the spherical correction
        dict(name="pixel_all_modes", kind="single", streams=32, layers=400, modes=241, L=120, surface="rough", ipss=1),
        # a short row of a batch file: the default streams, uneven layers, a few modes, every
        # surface kind, from host arrays to host arrays
        dict(name="row", kind="host", n=61, streams=24, layers=90, modes=8, L=60, surface="any", ipss=0),
        # a resident scene, executed again and again: uneven layers 50..400, 10 bands
        dict(name="scene", kind="plan", n=384, streams=32, layers=400, modes=32, L=120, surface="rough", ipss=0),
        # the same from host arrays to host arrays, the largest batch here
        dict(name="scene_host", kind="host", n=1024, streams=32, layers=400, modes=32, L=120, surface="rough", ipss=0),
        # a resident scene at the default 24 streams
        dict(name="scene_default_streams", kind="plan", n=500, streams=24, layers=150, modes=16, L=80,
             surface="rough", ipss=0),
        # Jacobians of a scene with respect to 200 layer depths, 200 albedos and the wind
        dict(name="jacobian", kind="jacobian", n=96, streams=32, layers=200, modes=32, L=120),
        # one step of a small retrieval: reflectance and its gradient through torch.autograd
        dict(name="retrieval", kind="autograd", n=7, streams=16, layers=40, modes=6, L=40),
        # coupled atmosphere-ocean pixel-bands: 400 air layers over 100 of water, a hydrosol of g = 0.92
        dict(name="ocean", kind="ocean", n=64, streams=32, layers=400, modes=16, L=120, water_layers=100, hydrosol=200),
        # one coupled pixel at the command line's defaults: pure sea water, 48 shared streams, modes 0..2
        dict(name="ocean_pixel", kind="ocean", n=1, streams=48, layers=40, modes=2, L=0, water_layers=0, hydrosol=0),
        # look-up tables on the command line's angle grid (35 x 144) for tabulated aerosols, spherical
        dict(name="lut", kind="lut", n=3, streams=32, layers=100, modes=16, L=80, step=2.5),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["single", "host", "plan", "plan", "jacobian", "autograd", "ocean", "lut"])
    streams = rng.choice([8, 12, 16, 20, 24, 24, 28, 31, 32, 32, 48])
    c = dict(kind=kind, streams=streams, layers=log(20, 400), modes=log(2, 32))
    c["L"] = max(2 * (c["modes"] // 2) + 8, log(20, 120))
    if kind in ("single", "host", "plan"):
        c["surface"] = rng.choice(["rough", "rough", "rough", "black", "any"])
        c["ipss"] = rng.choice([0, 0, 1])
    if kind in ("host", "plan"):
        c["n"] = log(2, 700)
        cost = c["n"] * c["modes"] * c["layers"] * streams ** 2
        c["n"] = max(2, min(c["n"], int(c["n"] * 700.0 * 32 * 200 * 32 ** 2 / cost)))
    elif kind == "jacobian":
        c["streams"] = rng.choice([8, 16, 24, 32])
        c["layers"] = log(20, 200)
        c["n"] = log(2, 90)
    elif kind == "autograd":
        c.update(streams=rng.choice([8, 12, 16, 24]), layers=log(10, 80), modes=log(2, 12), n=log(1, 16))
    elif kind == "ocean":
        c.update(streams=rng.choice([16, 24, 32, 32, 48]), modes=log(2, 16), n=log(1, 48), water_layers=log(20, 120),
                 hydrosol=rng.choice([0, 80, 200]))
        c["layers"] = log(20, 400)
        if c["streams"] == 48:
            c["n"] = min(c["n"], 4)
    elif kind == "lut":
        c.update(streams=rng.choice([16, 24, 32]), layers=log(20, 120), modes=log(2, 16), n=log(1, 4),
                 step=rng.choice([2.5, 5.0, 7.5]))
    return c


# ---------------------------------------------------------------- inputs
def _moments(g, L):
    """Henyey-Greenstein moments with Rayleigh-form polarisation scaled by 0.3."""
    l = np.arange(L + 1, dtype=np.float64)
    a = 2.0 * (1.0 - DEPOL) / (2.0 + DEPOL)
    gamma, alpha = np.zeros(L + 1), np.zeros(L + 1)
    gamma[2], alpha[2] = -0.3 * a * math.sqrt(1.5), 0.9 * a
    return (2.0 * l + 1.0) * g ** l, gamma, alpha, np.zeros(L + 1)


def _rows(case, seed):
    """The pixels of a case as plain numbers: geometry, wavelength, Rayleigh depth, wind, aerosol, layers."""
    rng = np.random.default_rng([int(seed) % (1 << 63), 7])
    n, nl = case.get("n", 1), case["layers"]
    uneven = case["kind"] in ("host", "plan")
    steps = [max(2, nl // 8), max(2, nl // 4), max(2, nl // 2), nl]
    kinds = {"rough": ["rough"], "black": ["black"], "any": ["rough", "black", "flat"]}[case.get("surface", "rough")]
    rows = []
    for i in range(n):
        wl = float(rng.choice(BANDS))
        rows.append(dict(
            sza=rng.uniform(0.0, 80.0 if uneven else 70.0), vza=rng.uniform(0.0, 70.0 if uneven else 60.0),
            raa=rng.uniform(0.0, 180.0), wl=wl, tau_r=0.0945 * (wl / 555.0) ** -4.08, wind=rng.uniform(1.0, 12.0),
            aod=math.exp(math.log(0.1) + 0.6 * rng.standard_normal()), ssa=rng.uniform(0.85, 0.99),
            g=rng.uniform(0.6, 0.8), layers=int(rng.choice(steps)) if uneven else nl, surface=kinds[i % len(kinds)]))
    return rows


def _native(case, rows):
    """The rows as the framework's records."""
    from ocrt_gb300 import _abi as A
    names = {"rough": "black_fresnel_ocean", "black": "black", "flat": "flat", "ocean": "ocean"}
    ocean = case["kind"] == "ocean"
    cases, opts, aers, mom = [], [], [], {}
    for r in rows:
        cases.append(A.default_case(surface=names["ocean" if ocean else r["surface"]], sza_deg=r["sza"], vza_deg=r["vza"],
                                    raa_deg=r["raa"], wavelength_nm=r["wl"], wind_speed=r["wind"], tau_r_input=r["tau_r"]))
        opts.append(A.default_opts(n_mu=case["streams"], n_layers=r["layers"], fourier_m_max=case["modes"],
                                   tau_r_source=A.TAU_R_FROM_INPUT, max_orders=1000, tolerance=1e-7,
                                   pssa=case.get("ipss", 1 if case["kind"] == "lut" else 0)))
        if case["L"] and case["kind"] == "lut":
            # a tabulated phase function beside the moments (the value kernel)
            th = np.concatenate([np.linspace(0.0, 10.0, 101), np.linspace(10.5, 180.0, 340)])
            p11 = (1 - r["g"] ** 2) / (1 + r["g"] ** 2 - 2 * r["g"] * np.cos(np.radians(th))) ** 1.5
            aers.append(A.AerosolHolder(r["aod"], r["ssa"], *_moments(r["g"], case["L"]),
                                        phase=(th, p11, -0.3 * p11, p11)))
        elif case["L"]:
            aers.append(A.AerosolHolder(r["aod"], r["ssa"], *_moments(r["g"], case["L"])))
    return cases, opts, aers or None


def prepare(case, seed):
    import ocrt_gb300 as og
    rows = _rows(case, seed)
    cases, opts, aers = _native(case, rows)
    st = dict(kind=case["kind"], cases=cases, opts=opts, aers=aers)
    if case["kind"] == "plan":
        st["plan"] = og.Plan(cases, opts, aers)
    elif case["kind"] == "jacobian":
        st["plan"] = og.Plan(cases, opts, aers, cot=np.broadcast_to(np.eye(3), (len(cases), 3, 3)).copy())
    elif case["kind"] == "autograd":
        from ocrt_gb300.autograd import layer_parameters
        dtau, ssa, wind = layer_parameters(cases, opts, aers)
        f1, f2, wgt = _perturbation(case, seed)
        st["params"] = [(dtau * f1).requires_grad_(), (ssa * f2).requires_grad_(), wind.requires_grad_()]
        st["weight"] = wgt
    elif case["kind"] == "ocean":
        from ocrt_gb300 import _abi as A
        rng = np.random.default_rng([int(seed) % (1 << 63), 11])
        st["oceans"] = []
        for i, c in enumerate(cases):
            wl = WATER_BANDS[i % len(WATER_BANDS)]
            c.wavelength_nm, c.tau_r_input = wl, 0.0945 * (wl / 555.0) ** -4.08
            bw = 0.0019 * (550.0 / wl) ** 4.32
            if case["hydrosol"]:
                a, b = rng.uniform(0.02, 0.5), rng.uniform(0.05, 1.0)
                st["oceans"].append(A.OceanHolder(a, bw, max(0.0, b - bw), _moments(0.92, case["hydrosol"]),
                                                  n_mu_water=case["streams"], m_max_water=case["modes"], depth_m=50.0,
                                                  n_layers_water=case["water_layers"], max_orders_water=1000))
            else:
                st["oceans"].append(A.OceanHolder(rng.uniform(0.02, 0.3), bw, n_mu_water=case["streams"],
                                                  m_max_water=case["modes"], n_layers_water=case["water_layers"]))
    elif case["kind"] == "lut":
        vza = np.arange(int(85.0 / case["step"]) + 1) * case["step"]
        raa = np.arange(int(360.0 / case["step"])) * case["step"]
        from ocrt_gb300 import _abi as A
        st["luts"] = [A.LutHolder(vza, raa) for _ in cases]
    return st


def _perturbation(case, seed):
    rng = np.random.default_rng([int(seed) % (1 << 63), 13])
    n, nt = case["n"], case["layers"]
    return (torch.from_numpy(rng.uniform(0.9, 1.1, (n, nt))), torch.from_numpy(rng.uniform(0.95, 1.0, (n, nt))),
            torch.from_numpy(rng.uniform(0.5, 1.5, (n, 3)) * rng.choice([-1.0, 1.0], (n, 3))))


_PLANES = {"rho": ("rho_I", "rho_Q", "rho_U"), "toa": ("I_TOA", "Q_TOA", "U_TOA"),
           "glint": ("rho_glint_direct_I", "rho_glint_direct_Q", "rho_glint_direct_U"),
           "transmittance": ("T_dir_dn", "T_diff_dn_hemi", "T_total_dn_hemi", "T_diff_dn_dir", "T_total_up_dir",
                             "T_sg_up_dir", "T_dir_up_view"),
           "column": ("tau_R_total", "kappa_ipss")}
_WATER = {"rho_atm": ("rho_atm_I", "rho_atm_Q", "rho_atm_U"), "rho_water": ("rho_water_I", "rho_water_Q", "rho_water_U"),
          "L_below": ("Lu_0minus_I", "Lu_0minus_Q", "Lu_0minus_U"), "L_above": ("Lu_0plus_I", "Lu_0plus_Q", "Lu_0plus_U"),
          "Rrs": ("Rrs_0plus_I", "Rrs_0plus_Q", "Rrs_0plus_U"), "rrs": ("rrs_0minus_I", "rrs_0minus_Q", "rrs_0minus_U"),
          "E": ("Ed_0minus", "Eu_0minus", "Ed_0plus", "Ed_0minus_direct", "Ed_0plus_direct"),
          "K": ("Kd_0minus", "Ku_0minus"), "water": ("tau_water", "depth_water_m")}


def _planes(res, names=_PLANES):
    out = {k: np.stack([np.asarray(res[f], dtype=np.float32) for f in v], axis=-1) for k, v in names.items()}
    out["converged"] = np.asarray(res["converged"], dtype=np.int32)
    return out


def run(state):
    import ocrt_gb300 as og
    kind, a = state["kind"], (state["cases"], state["opts"], state["aers"])
    if kind == "single":
        return _planes(og.solve_case(a[0][0], a[1][0], a[2][0] if a[2] else None))
    if kind == "host":
        return _planes(og.solve_batch(*a))
    if kind == "plan":
        state["plan"].execute()
        return _planes(state["plan"].results())
    if kind == "jacobian":
        state["plan"].execute()
        out = _planes(state["plan"].results())
        out.update({k: v.astype(np.float32) for k, v in state["plan"].gradients().items()})
        return out
    if kind == "autograd":
        from ocrt_gb300.autograd import sos_reflectance
        p = state["params"]
        rho = sos_reflectance(*p, *a)
        g = torch.autograd.grad((rho * state["weight"]).sum(), p)
        return {"rho": rho.detach().float(), "d_dtau": g[0].float(), "d_ssa": g[1].float(), "d_wind": g[2].float()}
    if kind == "ocean":
        res = og.solve_batch_ocean(a[0], a[1], state["oceans"], a[2])
        cols = {f: np.array([r[f] for r in res]) for f in res[0]}
        return {**_planes(cols), **_planes(cols, _WATER), "converged_water": cols["converged_water"].astype(np.int32)}
    res = og.solve_batch_lut(*a, state["luts"])
    out = _planes(res)
    for k in ("rho_I", "rho_Q", "rho_U", "T_diff_dn_dir", "T_sg_up_dir", "T_total_up_dir"):
        out["lut_" + k] = np.concatenate([x.out[k] for x in state["luts"]]).astype(np.float32)
    return out


def work(case):
    """Bytes: the input records and moments, the result records.  FLOPs: the source contraction
    alone (72 N^2 per level, mode and order; with six orders per mode, what a molecular and thin
    aerosol atmosphere needs at the least), twice over where a gradient is taken, three passes
    for the coupled solve."""
    n, N, M, K = case.get("n", 1), case["streams"], case["modes"] + 1, case["layers"] + 1
    if case["kind"] in ("host", "plan"):
        K = sum(max(2, case["layers"] // q) + 1 for q in (1, 2, 4, 8)) / 4.0
    mult = {"jacobian": 4, "autograd": 4}.get(case["kind"], 1)
    flops = n * M * K * 72.0 * N * N * 6 * mult
    out = 18 * 4 + 4
    if case["kind"] in ("jacobian", "autograd"):
        out += 3 * (2 * case["layers"] + 1) * 4
    if case["kind"] == "ocean":
        flops = n * M * 72.0 * N * N * 6 * (2 * K + max(case["water_layers"], 20) + 1)
        out += 26 * 4
    if case["kind"] == "lut":
        out += 6 * 4 * (int(85.0 / case["step"]) + 1) * int(360.0 / case["step"])
    return {"bytes": float(n * (96 + 88 + 32 * (case["L"] + 1) + out)), "flops": float(flops)}


# ---------------------------------------------------------------- the same in 64 bits
_F = torch.float64


def exact(case, seed):
    rows = _rows(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] in ("single", "host", "plan") and not case["ipss"] and case["surface"] != "any":
        if sum(r["layers"] for r in rows) * (case["modes"] + 1) * case["streams"] ** 2 > 3.6e9:
            return None
        rho, toa = torch.zeros(len(rows), 3, dtype=_F), torch.zeros(len(rows), 3, dtype=_F)
        for nt in sorted({r["layers"] for r in rows}):
            same = [i for i, r in enumerate(rows) if r["layers"] == nt]
            room = max(1, int(6e9 / (8 * (case["modes"] + 1) * (nt + 1) * 6 * (case["streams"] + 1))))
            for k in range(0, len(same), room):
                part = same[k:k + room]
                rho[part], toa[part] = (x.cpu() for x in _solve([rows[i] for i in part], case, dev)[:2])
        one = (lambda x: x[0].numpy()) if case["kind"] == "single" else (lambda x: x.numpy())
        return {"rho": one(rho), "toa": one(toa), "glint": None, "transmittance": None, "column": None, "converged": None}
    if case["kind"] == "autograd":
        if case["n"] * case["layers"] * case["modes"] > 3000:
            return None
        f1, f2, wgt = (x.to(dev) for x in _perturbation(case, seed))
        with torch.no_grad():
            dtau, ssa = _profile(rows, case, dev)
        p = [(dtau * f1).requires_grad_(), (ssa * f2).requires_grad_(),
             torch.tensor([r["wind"] for r in rows], dtype=_F, device=dev, requires_grad=True)]
        rho = _solve(rows, case, dev, p)[0]
        g = torch.autograd.grad((rho * wgt).sum(), p)
        return {"rho": rho.detach().cpu(), "d_dtau": g[0].cpu(), "d_ssa": g[1].cpu(), "d_wind": g[2].cpu()}
    return None


def _gauss(N):
    x, w = np.polynomial.legendre.leggauss(2 * N)
    return x[N:].copy(), w[N:].copy()


def _us62(z):
    """Column fraction above altitude z (km): US 1962 pressures, log-linear between the nodes, over gravity."""
    Z = torch.tensor([0.0, 11.0, 20.0, 32.0, 47.0, 51.0, 71.0, 84.852], dtype=_F, device=z.device)
    P = torch.tensor([101325.0, 22632.1, 5474.89, 868.019, 110.906, 66.9389, 3.95642, 0.3734], dtype=_F, device=z.device)
    s1 = math.sin(math.pi / 4) ** 2

    def grav(zz):
        return 9.780327 * (1.0 + 0.0053024 * s1 - 0.0000058) - 3.086e-3 * zz

    k = (torch.searchsorted(Z, z.contiguous(), right=True) - 1).clamp(0, 6)
    t = (z - Z[k]) / (Z[k + 1] - Z[k])
    p = torch.exp(torch.log(P[k]) + t * (torch.log(P[k + 1]) - torch.log(P[k])))
    q0, ft = 101325.0 / grav(0.0), 0.3734 / grav(84.852)
    raw = (p / grav(z)) / q0
    f = ((raw - ft / q0) / (1.0 - ft / q0)).clamp(0.0, 1.0)
    return torch.where(z <= 0, torch.ones_like(z), torch.where(z >= 84.852, torch.zeros_like(z), f))


def _mix(rows, case, dev):
    """Uniform optical-depth grid of rows of equal layer count: (total depth, x = aerosol and y =
    molecular scattering fraction per level)."""
    nt = rows[0]["layers"]
    col = lambda k: torch.tensor([r[k] for r in rows], dtype=_F, device=dev)[:, None]  # noqa: E731
    tr = col("tau_r")
    if not case["L"]:
        x = torch.zeros(len(rows), nt + 1, dtype=_F, device=dev)
        return tr, x, 1.0 - x
    ta, et = col("aod"), math.exp(-50.0)

    def aer(z):
        return torch.where(z >= 100.0, torch.zeros_like(z), ((torch.exp(-z / 2.0) - et) / (1.0 - et)).clamp(0.0, 1.0))

    tau = tr + ta
    h = tau * torch.arange(nt + 1, dtype=_F, device=dev) / nt
    lo, hi = torch.zeros_like(h), torch.full_like(h, 100.0)
    for _ in range(64):
        mid = 0.5 * (lo + hi)
        up = tr * _us62(mid) + ta * aer(mid) > h
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    z = 0.5 * (lo + hi)
    z[:, 0], z[:, nt] = 100.0, 0.0
    r, a = tr * _us62(z), ta * aer(z)
    r[:, 0] = a[:, 0] = 0.0
    x, y = torch.zeros_like(z), torch.ones_like(z)
    dr, da = r[:, 1:] - r[:, :-1], a[:, 1:] - a[:, :-1]
    x[:, 1:], y[:, 1:] = da * col("ssa") / (dr + da), dr / (dr + da)
    return tau, x, y


def _profile(rows, case, dev):
    tau, x, y = _mix(rows, case, dev)
    nt = rows[0]["layers"]
    return (tau / nt).expand(-1, nt).clone(), (x + y)[:, 1:].clone()


def _basis(L, m, x):
    """Normalised P_l^m and the spin-2 functions R_l^m, T_l^m at cosines x, degrees 0..L: [3, L + 1, len(x)]."""
    out = np.zeros((3, L + 1, x.size))
    P, R, T = out
    s2 = 1.0 - x * x
    l0 = max(2, m)
    if m == 0:
        P[0], P[1], P[2] = 1.0, x, 0.5 * (3 * x * x - 1)
        R[2] = 3.0 * s2 / (2.0 * math.sqrt(6.0))
    elif m == 1:
        P[1] = np.sqrt(0.5 * s2)
        P[2], R[2], T[2] = x * P[1] * math.sqrt(3.0), -0.5 * x * np.sqrt(s2), -0.5 * np.sqrt(s2)
    elif m <= L:
        d = math.exp(sum(0.5 * math.log((i + m) / i) - math.log(2.0) for i in range(1, m + 1)))
        sn = d * math.sqrt(m / (m + 1.0)) * math.sqrt((m - 1.0) / (m + 2.0))
        P[m], env = d * s2 ** (0.5 * m), s2 ** (0.5 * m - 1.0)
        R[m], T[m] = sn * (1 + x * x) * env, sn * 2 * x * env
    for l in range(l0, L):
        den = math.sqrt((l + m + 1.0) * (l - m + 1.0))
        P[l + 1] = ((2 * l + 1) * x * P[l] - math.sqrt((l + m) * (l - m)) * P[l - 1]) / den
        sc = (l + 1.0) * (2 * l + 1) / (math.sqrt((l + 3.0) * (l - 1.0)) * den)
        dc = math.sqrt((l + 2.0) * (l - 2.0) * (l + m) * (l - m)) / (l * (2.0 * l + 1))
        cc = 2.0 * m / (l * (l + 1.0))
        R[l + 1] = sc * (x * R[l] - cc * T[l] - dc * R[l - 1])
        T[l + 1] = sc * (x * T[l] - cc * R[l] - dc * T[l - 1])
    return out


def _pi(b):
    """Stokes matrices [[P, 0, 0], [0, R, -T], [0, -T, R]] of a basis [3, L + 1, n]: [n, 3, L + 1, 3]."""
    P, R, T = b.transpose(0, 2, 1)
    z = np.zeros_like(P)
    return np.stack([np.stack([P, z, z], -1), np.stack([z, R, -T], -1), np.stack([z, -T, R], -1)], 1)


def _mueller(mo, mi, phi, s2, lam, nw=1.34):
    """Cox-Munk reflection matrix of facets with slope variance s2 and shadowing lam; mo outgoing
    and mi incoming cosines, phi the azimuth: [..., 3, 3]."""
    so, si = torch.sqrt(1 - mo * mo), torch.sqrt(1 - mi * mi)
    cT = (-mo * mi + so * si * torch.cos(phi)).clamp(-1, 1)
    A = (mo + mi) ** 2
    B = (so - si) ** 2 + 4 * so * si * torch.sin(0.5 * phi) ** 2
    cw, tan2 = 0.5 * torch.sqrt(A + B), B / A
    cb2 = A / (A + B)
    u1, v1 = (mo + mi * cT) / si, so * torch.sin(phi)
    u2, v2 = (-mi - mo * cT) / so, si * torch.sin(phi)
    n1, n2 = u1 * u1 + v1 * v1, u2 * u2 + v2 * v2
    a1, b1, a2, b2 = (u1 * u1 - v1 * v1) / n1, 2 * u1 * v1 / n1, (u2 * u2 - v2 * v2) / n2, 2 * u2 * v2 / n2
    mt = torch.sqrt(1 - (1 - cw * cw) / nw ** 2)
    rs, rp = (cw - nw * mt) / (cw + nw * mt), (nw * cw - mt) / (nw * cw + mt)
    f0, f1, f8 = 0.5 * (rs * rs + rp * rp), 0.5 * (rp * rp - rs * rs), rs * rp
    brdf = torch.exp(-tan2 / s2) / (math.pi * s2 * (1 + lam) * 4 * mi * mo * cb2 * cb2)
    M11, M12, M21, M22 = f0 * a1, -f0 * b1, f8 * b1, f8 * a1
    R = [f0 + 0 * a1, f1 * a1, -f1 * b1, a2 * f1, a2 * M11 - b2 * M21, a2 * M12 - b2 * M22,
         b2 * f1, b2 * M11 + a2 * M21, b2 * M12 + a2 * M22]
    return torch.stack([e * brdf for e in torch.broadcast_tensors(*R)], -1).unflatten(-1, (3, 3))


def _shadow(mu, s2):
    nu = mu / torch.sqrt(((1 - mu * mu)).clamp_min(1e-20) * s2)
    lam = 0.5 * (torch.exp(-nu * nu) / (nu * math.sqrt(math.pi)) - torch.special.erfc(nu))
    return torch.where((nu > 20.0) | (mu >= 1 - 1e-10), torch.zeros_like(lam), lam)


def _surface(ring, mu0, s2, N, M):
    """Fourier kernels of one pixel: [M + 1, ring slots, N + 1 (Gauss nodes and the sun), 3, 3]."""
    half = 512
    phi = (torch.arange(half, dtype=_F, device=ring.device) + 0.5) * math.pi / half
    inc = torch.cat([ring[:N], mu0[None]])
    lam = _shadow(ring, s2)[:, None, None] + _shadow(inc, s2)[None, :, None]
    R = _mueller(ring[:, None, None], inc[None, :, None], phi, s2, lam)
    m = torch.arange(M + 1, dtype=_F, device=ring.device)
    C, S = torch.cos(m[:, None] * phi) * (2.0 / half), torch.sin(m[:, None] * phi) * (2.0 / half)
    C, S = torch.cat([C[:1] * 0.5, C[1:]]), torch.cat([S[:1] * 0.5, S[1:]])
    flip = torch.ones(M + 1, 1, 1, dtype=_F, device=ring.device)
    flip[1:] = -1.0
    c, s = torch.einsum("mq,oiqab->moiab", C, R), torch.einsum("mq,oiqab->moiab", S, R)
    r0 = torch.stack([c[..., 0, 0], c[..., 0, 1], flip * s[..., 0, 2]], -1)
    r1 = torch.stack([c[..., 1, 0], c[..., 1, 1], flip * s[..., 1, 2]], -1)
    r2 = torch.stack([s[..., 2, 0], s[..., 2, 1], c[..., 2, 2]], -1)
    return torch.stack([r0, r1, r2], -2)


def _solve(rows, case, dev, params=None):
    """TOA reflectance [P, 3] and radiance of pixels with equal layer counts, FP64: the modes'
    successive orders, each summed until it adds 1e-10 of its total at the output levels."""
    P, N, M, nt = len(rows), case["streams"], case["modes"], rows[0]["layers"]
    t = lambda v: torch.as_tensor(np.asarray(v), dtype=_F, device=dev)  # noqa: E731
    gm, gw = _gauss(N)
    rough = rows[0].get("surface", "rough") == "rough"
    mu0n, muvn = np.cos(np.radians([r["sza"] for r in rows])), np.cos(np.radians([r["vza"] for r in rows]))
    mu0, muv = t(mu0n), t(muvn)
    ring = torch.cat([t(gm).expand(P, N), muv[:, None]], 1)
    tau, x, y = _mix(rows, case, dev)
    wind = t([r["wind"] for r in rows])
    h = tau * torch.arange(nt + 1, dtype=_F, device=dev) / nt
    if params is not None:
        dtau, ssa, wind = params
        h = torch.cat([torch.zeros(P, 1, dtype=_F, device=dev), torch.cumsum(dtau, 1)], 1)
        w0 = (x + y)[:, 1:]
        x = torch.cat([x[:, :1], x[:, 1:] * ssa / w0], 1)
        y = torch.cat([y[:, :1], y[:, 1:] * ssa / w0], 1)
        tau = h[:, -1:]
    ch = 0.5 * torch.exp(-h / mu0[:, None])
    # transport weights of every layer and ring slot
    xx = ((h[:, 1:] - h[:, :-1])[:, :, None] / ring[:, None, :])[:, :, None, :]
    T = torch.exp(-xx)
    G = -torch.expm1(-xx) / xx - T
    Ca, Cb = 0.5 * (1 - T - G), 0.5 * G
    # phase operators Z^m: outgoing [h (up, down), s, ring], incoming [h, s, Gauss], weights folded in; solar columns
    a = 2.0 * (1 - DEPOL) / (2 + DEPOL)
    mol = np.zeros((3, 3, 3))
    mol[0, 0, 0], mol[2, 0, 0], mol[2, 0, 1], mol[2, 1, 0], mol[2, 1, 1] = 1.0, 0.5 * a, -a * 1.5 ** 0.5, -a * 1.5 ** 0.5, 3 * a
    L = max(case["L"], 2)
    mats = []
    for r in rows:
        B = np.zeros((L + 1, 3, 3))
        if case["L"]:
            be, ga, al, ze = _moments(r["g"], case["L"])
            B[:, 0, 0], B[:, 0, 1], B[:, 1, 0], B[:, 1, 1], B[:, 2, 2] = be, ga, ga, al, ze
        mats.append(B)
    Bl, w2 = t(np.stack(mats)), t(np.tile(gw, 6))
    ops = []
    for m in range(M + 1):
        pg = _pi(_basis(L, m, np.concatenate([gm, -gm])))
        pv = _pi(_basis(L, m, np.concatenate([muvn, -muvn, -mu0n])))
        pg, pv = t(pg).reshape(2, N, 3, L + 1, 3), t(pv).reshape(3, P, 3, L + 1, 3)
        out = torch.cat([pg.permute(0, 2, 1, 3, 4).expand(P, 2, 3, N, L + 1, 3),
                         pv[:2].permute(1, 0, 2, 3, 4)[:, :, :, None]], 3)                  # [P, 2, 3, N + 1, L + 1, 3]
        inc = pg.permute(0, 2, 1, 3, 4).reshape(6 * N, -1)
        za = torch.einsum("phsgla,plab->phsglb", out, Bl).reshape(P, 6 * (N + 1), -1)
        sun = pv[2][:, 0].reshape(P, -1, 1)
        zm = torch.zeros(P, 6 * (N + 1), 1, dtype=_F, device=dev)
        om, sm = torch.zeros(P, 6 * (N + 1), 6 * N, dtype=_F, device=dev), zm
        if m <= 2:
            zo = torch.einsum("phsgla,lab->phsglb", out[..., :3, :], t(mol)).reshape(P, 6 * (N + 1), -1)
            om = zo @ pg[..., :3, :].permute(0, 2, 1, 3, 4).reshape(6 * N, -1).T * w2
            sm = zo @ pv[2][:, 0, :3].reshape(P, -1, 1)
        ops.append((za @ inc.T * w2, (za @ sun)[..., 0], om, sm[..., 0]))
    oa, sa = torch.stack([o[0] for o in ops], 1), torch.stack([o[1] for o in ops], 1)
    om, sm = torch.stack([o[2] for o in ops[:3]], 1), torch.stack([o[3] for o in ops], 1)
    # surface
    s2 = 0.003 + 0.00512 * wind
    mm = torch.arange(M + 1, dtype=_F, device=dev)
    fac = torch.where(mm == 0, 2.0, 1.0) * math.pi
    seed = torch.zeros(P, M + 1, nt + 1, 3, N + 1, dtype=_F, device=dev)
    if rough:
        R = torch.stack([_surface(ring[p], mu0[p], s2[p], N, M) for p in range(P)])
        bc_op = torch.einsum("pmgiab,i,m->pmagbi", R[:, :, :, :N], t(gm * gw), fac)
        att = torch.exp(-(tau - h)[:, :, None] / ring[:, None, :])
        seed = torch.einsum("m,p,pkg,pmga->pmkag", 0.5 * fac, mu0 * torch.exp(-tau[:, 0] / mu0), att, R[:, :, :, N, :, 0])

    def scan(J, bc):
        up, dn = [bc], [torch.zeros_like(bc)]
        for k in range(nt - 1, -1, -1):
            up.append(T[:, None, k] * up[-1] + Ca[:, None, k] * J[:, :, k, 0] + Cb[:, None, k] * J[:, :, k + 1, 0])
        for k in range(1, nt + 1):
            dn.append(T[:, None, k - 1] * dn[-1] + Ca[:, None, k - 1] * J[:, :, k, 1] + Cb[:, None, k - 1] * J[:, :, k - 1, 1])
        return torch.stack([torch.stack(up[::-1], 2), torch.stack(dn, 2)], 3)               # [P, m, k, 2, 3, N + 1]

    shape = (P, M + 1, nt + 1, 2, 3, N + 1)
    J = ch[:, None, :, None] * (x[:, None, :, None] * sa[:, :, None] + y[:, None, :, None] * sm[:, :, None])
    zero = torch.zeros(P, M + 1, 3, N + 1, dtype=_F, device=dev)
    F = scan(J.reshape(shape), zero)
    F = torch.cat([(F[:, :, :, 0] + seed)[:, :, :, None], F[:, :, :, 1:]], 3)
    ends = F[:, :, [0, nt]]
    live = torch.ones(P, M + 1, dtype=torch.bool, device=dev)
    for _ in range(999):
        V = F[..., :N].reshape(P, M + 1, nt + 1, 6 * N)
        J = x[:, None, :, None] * (V @ oa.transpose(-1, -2))
        k = min(3, M + 1)
        Jm = y[:, None, :, None] * (V[:, :k] @ om.transpose(-1, -2))
        J = torch.cat([J[:, :k] + Jm, J[:, k:]], 1)
        bc = torch.einsum("pmagbi,pmbi->pmag", bc_op, F[:, :, nt, 1, :, :N]) if rough else zero
        F = scan(J.reshape(shape), bc) * live[:, :, None, None, None, None]
        ends = ends + F[:, :, [0, nt]]
        big = F.detach().abs().amax((2, 3, 4, 5))
        live = live & ~(big < 1e-10 * ends.detach().abs().amax((2, 3, 4, 5)))
        if not bool(live.any()):
            break
    view = ends[:, :, 0, 0, :, N] - seed[:, :, 0, :, N]
    phi = t(np.radians([r["raa"] for r in rows]) + math.pi)
    e = torch.where(mm == 0, 1.0, 2.0)
    c, s = e * torch.cos(mm * phi[:, None]), e * torch.sin(mm * phi[:, None])
    toa = torch.stack([(c * view[..., 0]).sum(1), (c * view[..., 1]).sum(1), (s * view[..., 2]).sum(1)], 1)
    rho = toa / mu0[:, None]
    if rough:
        lam = _shadow(mu0, s2) + _shadow(muv, s2)
        Rg = _mueller(muv, mu0, t(np.radians([r["raa"] - 180.0 for r in rows])), s2, lam)
        g = math.pi * Rg[:, :, 0] * torch.exp(-tau[:, 0] / mu0 - tau[:, 0] / muv)[:, None]
        rho = rho + g * t([1.0, 1.0, -1.0])
    return rho, toa
