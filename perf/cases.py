"""What a user of this framework has it do, as timed cases over its public
entry points.

Kinds of cases (``case["kind"]``):

* ``step``: advection steps of one device-resident state (``DeviceState``) from
  a checkpoint: the state is put back and advanced ``steps`` steps, as runs that
  start from the same spun-up state do.  FP64 (the default) and mixed
  precision, per-pair and thinned draws, both solutes, with and without
  collisions, fresh and raining clouds.
* ``batch``: one step of an ensemble (``BatchState``), which goes on from where
  the last pass left it.
* ``dropin``: ``integrate_adv_step_np`` on the reference's NumPy arrays, in
  place, call after call.
* ``box``: the collision box model (``simulate_collisions``), Golovin kernel or
  a tabulated collection efficiency with Beard velocities.
* ``adjoint``: objective and gradients of a recorded run (``StepModel``).

Raining states carry drops of 60 to 400 um in every cell of the cloud and below
it, and their SIPs lie in memory in any order, as after an hour of motion;
fresh states are ordered by cell, as the initialisation leaves them.
"""
import math

import numpy as np
import torch

from lacmopy_gb300 import BatchState, DeviceState, adjoint, collision, integration, synthetic

F64 = torch.float64


def listed():
    step = dict(kind="step", uneven=0, collisions=True, solute="AS", kernel="Long_Bott",
                draws="philox", precision="fp64", rain=False)
    return [
        # the smallest call: a test-sized grid, where launches and their gaps count
        dict(step, name="small_fp64", nx=12, nz=10, spc=16, uneven=8, steps=10),
        # the reference's own case (75 x 75 cells, 64 SIPs per cell), default precision and draws
        dict(step, name="icmw_fp64", nx=75, nz=75, spc=64, steps=2),
        # the two hours of spin-up before it (128 SIPs per cell, no collisions, no gravity)
        dict(step, name="spinup_fp64", nx=75, nz=75, spc=128, steps=2, collisions=False),
        # odd sizes, sea-salt aerosol, uneven cells, a raining cloud
        dict(step, name="nacl_rain_fp64", nx=101, nz=63, spc=85, uneven=64, steps=2, solute="NaCl",
             kernel="Hall_Bott", draws="thinned", rain=True),
        # one long mixed-precision run of the same case in its raining hour
        dict(step, name="icmw_rain_mixed", nx=75, nz=75, spc=128, steps=5, precision="mixed",
             rain=True),
        # the ensemble of 64 seeds (Hall kernel, 32 to 256 SIPs per cell), fresh
        dict(kind="batch", name="ensemble64_mixed", members=64, nx=75, nz=75, spc=144, uneven=112,
             kernel="Hall_Bott", draws="thinned", precision="mixed", rain=False),
        # a smaller ensemble in its raining hour
        dict(kind="batch", name="ensemble12_rain_mixed", members=12, nx=75, nz=75, spc=144,
             uneven=112, kernel="Hall_Bott", draws="thinned", precision="mixed", rain=True),
        # the reference's driver with the step function swapped: NumPy arrays in and out
        dict(kind="dropin", name="dropin_mixed", nx=75, nz=75, spc=144, uneven=112,
             kernel="Hall_Bott", draws="thinned", precision="mixed", rain=False),
        # box models: 5000 SIPs with the Golovin kernel, 2980 with Hall efficiencies
        dict(kind="box", name="golovin_box", method="golovin", sips=5000, growth=1.0, steps=4),
        dict(kind="box", name="hall_box", method="Hall_Bott", sips=2980, growth=1.5, steps=4),
        # gradients: of condensation and advection, and with the collections of a raining run
        dict(kind="adjoint", name="adjoint", nx=75, nz=75, spc=128, uneven=0, steps=2,
             collisions=False, rain=False),
        dict(kind="adjoint", name="adjoint_rain", nx=40, nz=31, spc=40, uneven=16, steps=6,
             collisions=True, rain=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, most, nx_max=150):
    """Grid and SIPs per cell with at most ``most`` SIPs in all."""
    while True:
        nx, nz = _log_int(rng, 8, nx_max), _log_int(rng, 8, nx_max)
        spc = _log_int(rng, 12, 200)
        if nx * nz * spc <= most:
            return dict(nx=nx, nz=nz, spc=spc, uneven=rng.choice((0, spc // 2, (3 * spc) // 4)))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "batch", "batch", "dropin", "box", "box",
                       "adjoint"))
    if kind == "step":
        precision = rng.choice(("fp64", "fp64", "mixed"))
        c = dict(_sizes(rng, 1000000), kind=kind, steps=rng.randint(1, 6), precision=precision,
                 collisions=rng.random() < 0.75, solute=rng.choice(("AS", "AS", "NaCl")),
                 kernel=rng.choice(("Long_Bott", "Hall_Bott")),
                 draws=rng.choice(("philox", "thinned")), rain=rng.random() < 0.5)
        return c
    if kind == "batch":
        c = _sizes(rng, 900000, 90)
        members = max(2, min(64, _log_int(rng, 2, 64), 40000000 // (c["nx"] * c["nz"] * c["spc"])))
        return dict(c, kind=kind, members=members, kernel=rng.choice(("Long_Bott", "Hall_Bott")),
                    draws=rng.choice(("thinned", "thinned", "philox")), precision="mixed",
                    rain=rng.random() < 0.5)
    if kind == "dropin":
        return dict(_sizes(rng, 900000), kind=kind, kernel=rng.choice(("Long_Bott", "Hall_Bott")),
                    draws=rng.choice(("philox", "thinned")),
                    precision=rng.choice(("fp64", "mixed")), rain=rng.random() < 0.5)
    if kind == "box":
        method = rng.choice(("golovin", "Hall_Bott", "Long_Bott"))
        return dict(kind=kind, method=method, growth=rng.uniform(1.0, 2.5),
                    sips=_log_int(rng, 60, 7000 if method == "golovin" else 4000),
                    steps=rng.randint(2, 6))
    collisions = rng.random() < 0.5
    return dict(_sizes(rng, 100000 if collisions else 700000, 90), kind=kind,
                steps=rng.randint(1, 4), collisions=collisions, rain=collisions)


# ---------------------------------------------------------------------------
# physical constants and fits (the reference model's; masses in fg, radii in um)
R_V, R_D, C_PD = 461.53, 287.06, 1004.71
KAPPA = R_D / C_PD
KF = 1.0 / (1.0 - KAPPA)
KF2 = -KAPPA * KF
EPS_GC = R_D / R_V
HEAT_RV = (1906 - R_V) / (C_PD - R_D)
FOUR_THIRDS_PI = 4.0 * math.pi / 3.0
RHO_WATER = (1.00013502e+03, -4.68112708e-03, 2.72389977e+02)
RHO_NACL = (7.619443952135e+02, 1.021264281453e+03, 1.828970151543, 2.405352122804e+02,
            -1.080547892416, -3.492805028749e-03)
RHO_AS = tuple(v / 997.1 for v in (1.024E1, -5.036E1, 592., 997.1))
SIGMA_AS, SIGMA_NACL = 2.362E-3 / 132.14E-3 / 0.072, 1.62E-3 / 58.4428E-3 / 0.072
ACT_AS = (1.412, -2.336, 3.113E-1, -2.715E-1, 1.0)
ACT_NACL = (1.518E1, -1.158E1, 8.642E-1, -6.366E-1, 1.0)
W_MAX_INV = 1. / 0.78
T_A0 = 289.
_ALPHA = C_PD * 0.7142857142857143 + 0.5 * R_D
C_ALPHA = (1.0E6 * math.sqrt(2.0 * math.pi * R_D * T_A0) / _ALPHA,
           0.5E6 * math.sqrt(2.0 * math.pi * R_D / T_A0) / _ALPHA)
C_BETA = (1.0E6 * math.sqrt(2.0 * math.pi * 18.015E-3 / (8.3144598 * T_A0)) / 0.0415, -0.5 / T_A0)


def _poly(par, x):
    r = par[0] * x + par[1]
    for a in par[2:]:
        r = r * x + a
    return r


def _deriv(par):
    n = len(par) - 1
    return tuple(par[k] * (n - k) for k in range(n))


def _ambient(Th, rv, rho_d, p_ref=1.0E5):
    """The cell quantities that follow from Theta, r_v and the dry density."""
    pdr = (rho_d * Th * R_D / p_ref) ** KF
    T = Th * pdr ** KAPPA
    p = pdr * p_ref * (1.0 + rv / EPS_GC)
    e_s = 2.53E11 * torch.exp(-5420.0 / T)
    tau = 1.0 - T / 647.096
    return dict(T=T, p=p, e_s=e_s, S=rho_d * rv * T * R_V / e_s,
                K=4.1868E-3 * (5.69 + 0.017 * (T - 273.15)), D_v=4.01218E-5 * T ** 1.94 / p,
                L_v=1.0E3 * (2500.82 - 2.358 * (T - 273.0)),
                sig_w=0.2358 * tau ** 1.256 * (1.0 - 0.625 * tau),
                rho_w=RHO_WATER[0] + RHO_WATER[1] * (T - RHO_WATER[2]) ** 2,
                mu=1.458E-6 * T ** 1.5 / (T + 110.4), rho_f=rho_d * (1.0 + rv))


# ---------------------------------------------------------------------------
# inputs
def _base(case, seed):
    """Grid, profiles, parameters and efficiency table of the case (host)."""
    return synthetic.make_icmw_state(Nx=case["nx"], Nz=case["nz"], no_spcm=(1, 1), seed=seed,
                                     kernel_type=case.get("kernel", "Long_Bott"),
                                     r_tot=8.5E-3 if case["nz"] >= 40 else 12.0E-3)


def _members(case, seed, M):
    """M states of the case on the GPU.  Each attribute of all members lies in
    one buffer; a member's arrays are its slices.  Returns (dicts, buffers)."""
    base = _base(case, seed)
    nx, nz, spc, un = case["nx"], case["nz"], case["spc"], case["uneven"]
    C = nx * nz
    dx, dz = base["grid_steps"]
    V = float(base["grid_volume_cell"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=F64)  # noqa: E731
    gsf0 = torch.from_numpy(base["grid_scalar_fields"]).cuda().reshape(10, C)
    # grid fields of every member: small deviations of Theta and r_v
    noise = torch.randn(2, M, C, generator=g, device="cuda", dtype=F64)
    Th = gsf0[2] + 0.01 * noise[0]
    rv = gsf0[4] * (1.0 + 1e-4 * noise[1])
    rho_d = gsf0[3].expand(M, C)
    a = _ambient(Th, rv, rho_d)
    rv = rv / a["S"] * torch.clamp(a["S"], max=1.0015)
    a = _ambient(Th, rv, rho_d)
    gsf = torch.stack([a["T"], a["p"], Th, rho_d, rv, gsf0[5].expand(M, C), a["S"], a["e_s"],
                       gsf0[8].expand(M, C), gsf0[9].expand(M, C)], 1).contiguous()
    gmp = torch.stack([a["K"], a["D_v"], a["L_v"], a["sig_w"], C_PD * (1 + 0.897 * rv), a["mu"],
                       a["rho_f"]], 1).contiguous()
    # SIPs, cell after cell: two aerosol modes, stratified in the log of the dry radius
    # (their counts in the cells are shuffled by the seed, their number is the case's)
    fixed = torch.Generator(device="cuda").manual_seed(spc * 1000003 + C)
    cnt = torch.randint(max(2, spc - un), spc + un + 1, (M, C), generator=fixed, device="cuda")
    cnt = torch.gather(cnt, 1, torch.argsort(rand(M, C), dim=1))
    n_m = cnt.sum(1).tolist()
    cnt = cnt.reshape(-1)
    N = sum(n_m)
    mc = torch.repeat_interleave(torch.arange(M * C, device="cuda"), cnt, output_size=N)
    n = cnt[mc]
    rank = torch.arange(N, device="cuda") - (torch.cumsum(cnt, 0) - cnt)[mc]
    n0 = torch.clamp((n * 26 + 32) // 64, min=1)
    big = rank >= n0
    n_k = torch.where(big, n - n0, n0)
    r_k = torch.where(big, rank - n0, rank)
    del rank, n, n0
    mu = torch.where(big, math.log(0.075), math.log(0.02)).to(F64)
    sg = torch.where(big, math.log(1.6), math.log(1.4)).to(F64)
    conc = torch.where(big, 40.0E6, 60.0E6).to(F64)
    width = 7.0 * sg / n_k
    ln_R = mu - 3.5 * sg + (r_k + rand(N)) * width
    xi = conc * V * width * torch.exp(-0.5 * ((ln_R - mu) / sg) ** 2) / (math.sqrt(2 * math.pi) * sg)
    R_s = torch.exp(ln_R)
    del mu, sg, conc, width, ln_R, r_k, n_k, big
    rho_s = 1774.0 if case.get("solute", "AS") == "AS" else 2163.0
    m_s = FOUR_THIRDS_PI * rho_s * R_s ** 3
    # haze in equilibrium with its cell, activated drops that share the cell's liquid water
    act_par = ACT_AS if case.get("solute", "AS") == "AS" else ACT_NACL
    w_top = 0.78 if case.get("solute", "AS") == "AS" else 0.25
    Sc = torch.clamp(a["S"].reshape(-1), 0.5, 0.999)
    lo, hi = torch.zeros_like(Sc), torch.full_like(Sc, w_top)
    for _ in range(50):
        mid = 0.5 * (lo + hi)
        up = _poly(act_par, mid) > Sc
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    w_s = torch.clamp(0.5 * (lo + hi), 0.02, w_top * 0.98)[mc]
    m_w = m_s * (1.0 / w_s - 1.0)
    c = mc % C
    r_l = torch.clamp((8.5E-3 if nz >= 40 else 12.0E-3) - gsf0[4], min=0.0)
    r_l = torch.where(a["S"] > 0.9995, r_l, torch.zeros_like(r_l)).reshape(-1)[mc]
    cloudy = r_l > 1e-5
    act = cloudy & (R_s > 0.035)
    drop = r_l * gsf0[3][c] / 40.8E6 * 1e18 * (0.5 + rand(N))
    m_w = torch.where(act, torch.maximum(drop, m_w), m_w)
    driz = act & (rand(N) < 0.03)
    R_d = 25.0 + 35.0 * rand(N)
    m_w = torch.where(driz, FOUR_THIRDS_PI * 1000.0 * R_d ** 3, m_w)
    xi = torch.where(driz, torch.exp(math.log(1e4) + math.log(1e2) * rand(N)), xi)
    fall = torch.where(driz, 1.2E8 * (R_d * 1e-6) ** 2, torch.zeros_like(m_w))
    if case["rain"]:
        rain = rand(N) < 0.008
        R_r = 60.0 * torch.exp(math.log(400.0 / 60.0) * rand(N))
        m_r = FOUR_THIRDS_PI * 1000.0 * R_r ** 3
        m_w = torch.where(rain, m_r, m_w)
        xi = torch.where(rain, 2.0E16 * rand(N) / m_r + 1.0, xi)
        fall = torch.where(rain, 8.0E-3 * R_r, fall)
        del rain, R_r, m_r
    del R_s, w_s, r_l, drop, driz, R_d, act, cloudy
    ci, cj = c // nz, c % nz
    x = (ci + rand(N)) * dx
    z = (cj + rand(N)) * dz
    gv = torch.from_numpy(base["grid_velocity"]).cuda()
    u = 0.5 * (gv[0, ci, cj] + gv[0, ci + 1, cj])
    w = 0.5 * (gv[1, ci, cj] + gv[1, ci, cj + 1]) - fall
    del fall
    member = mc // C
    if case["rain"]:   # SIPs in any order within their member
        order = torch.argsort(member + rand(N))
        x, z, u, w, m_w, m_s, xi, ci, cj = (t[order] for t in (x, z, u, w, m_w, m_s, xi, ci, cj))
    pad = lambda k: (k + 63) // 64 * 64  # noqa: E731
    tot = sum(pad(k) for k in n_m)
    buf = {k: torch.zeros(f * tot, dtype=F64, device="cuda")
           for k, f in (("pos", 2), ("vel", 2), ("rel_pos", 2), ("m_w", 1), ("m_s", 1), ("xi", 1),
                        ("T_p", 1))}
    buf["grid"], buf["mat"] = gsf, gmp
    buf["dml"] = torch.zeros(M, C, dtype=F64, device="cuda")
    buf["water"] = torch.zeros(M, 2, dtype=F64, device="cuda")
    buf["no_cols"] = torch.zeros(M, 2, dtype=torch.int64, device="cuda")
    Tc = a["T"].reshape(-1)
    out, s, o = [], 0, 0
    for m in range(M):
        k = n_m[m]
        cut = lambda name, f=1: buf[name][f * o:f * o + f * k]  # noqa: E731
        st = dict(base)
        ii, jj, sl = ci[s:s + k], cj[s:s + k], slice(s, s + k)
        pos = cut("pos", 2).view(2, k)
        pos[0], pos[1] = x[sl], z[sl]
        vel = cut("vel", 2).view(2, k)
        vel[0], vel[1] = u[sl], w[sl]
        rel = cut("rel_pos", 2).view(2, k)
        rel[0], rel[1] = pos[0] / dx - ii, pos[1] / dz - jj
        for name, t in (("m_w", m_w), ("m_s", m_s), ("xi", xi)):
            cut(name).copy_(t[sl])
        cut("T_p").copy_(Tc[m * C + ii * nz + jj])
        st.update(pos=pos, vel=vel, rel_pos=rel, m_w=cut("m_w"), m_s=cut("m_s"), xi=cut("xi"),
                  T_p=cut("T_p"), cells=torch.stack([ii, jj]),
                  active_ids=torch.ones(k, dtype=torch.uint8, device="cuda"),
                  grid_scalar_fields=gsf[m].view(10, nx, nz), grid_mat_prop=gmp[m].view(7, nx, nz),
                  delta_m_l=buf["dml"][m].view(nx, nz), water_removed=buf["water"][m, :1],
                  no_cols=buf["no_cols"][m], id_list=None,
                  solute_type=case.get("solute", "AS"))
        if not case.get("collisions", True):
            st["act_collisions"] = False
        if case["kind"] == "step" and not case["collisions"]:   # the reference's spin-up
            st.update(act_relaxation=False, g_set=0.0)
        out.append(st)
        s += k
        o += pad(k)
    return out, buf


def _host(st):
    """The state as the reference's NumPy arrays."""
    h = {k: (v.cpu().numpy().copy() if isinstance(v, torch.Tensor) else v) for k, v in st.items()}
    h["active_ids"] = h["active_ids"].astype(bool)
    h["id_list"] = np.arange(h["m_w"].size)
    return h


def _box(case, seed):
    """SIPs of a box model with exponential masses: one SIP per bin of the log
    mass; ``growth`` scales the mean radius (a later time of the run)."""
    rng = np.random.default_rng(seed)
    n = case["sips"]
    m_mean = FOUR_THIRDS_PI * 1000.0 * (9.3 * case["growth"]) ** 3
    edges = np.exp(np.linspace(math.log(2e-4 * m_mean), math.log(20.0 * m_mean), n + 1))
    masses = edges[:-1] + rng.random(n) * np.diff(edges)
    xis = 1e-3 * 1e18 / m_mean * np.exp(-masses / m_mean) / m_mean * np.diff(edges)
    xis = xis + 1.0
    radii = (masses / (FOUR_THIRDS_PI * 1000.0)) ** (1.0 / 3.0)
    return xis, masses, radii


def prepare(case, seed):
    kind = case["kind"]
    if kind == "box":
        xis, masses, radii = _box(case, seed)
        s = dict(kind=kind, steps=case["steps"], seed=seed, xis=xis, masses=masses)
        if case["method"] == "golovin":
            return dict(s, method=None, name="Golovin", kernel=None)
        b = _base(dict(nx=8, nz=8, kernel=case["method"]), 1)
        vel = np.zeros_like(radii)
        collision.update_velocity_Beard(vel, radii)
        return dict(s, method="Ecol_grid_R", name=case["method"], radii=radii, vel=vel,
                    rho=np.full_like(radii, 1000.0),
                    kernel=(b["E_col_grid"], b["no_kernel_bins"], b["R_kernel_low_log"],
                            b["bin_factor_R_log"]))
    if kind == "adjoint":
        st = _host(_members(case, seed, 1)[0][0])
        model = adjoint.StepModel(st, case["steps"])
        m_s = model.m_s0.clone().requires_grad_()
        kappa = torch.tensor(0.6, dtype=F64, device="cuda", requires_grad=True)
        flux = torch.tensor(1.0, dtype=F64, device="cuda", requires_grad=True)
        return dict(kind=kind, model=model, m_s=m_s, kappa=kappa, flux=flux,
                    weights=model.lwp_weights() + 100.0 * model.rain_weights())
    if kind == "dropin":
        st = _host(_members(case, seed, 1)[0][0])
        return dict(kind=kind, st=st, seed=seed, draws=case["draws"], precision=case["precision"],
                    col_step=0)
    if kind == "batch":
        sts, buf = _members(case, seed, case["members"])
        b = BatchState(sts, [seed + 1 + m for m in range(len(sts))], precision=case["precision"],
                       draws=case["draws"])
        return dict(kind=kind, batch=b, buf=buf)
    sts, buf = _members(case, seed, 1)
    ds = DeviceState(sts[0], draws=case["draws"], seed=seed, precision=case["precision"])
    live = [buf[k] for k in ("pos", "vel", "rel_pos", "m_w", "m_s", "xi", "T_p", "grid", "mat",
                             "dml", "water", "no_cols")] + [ds.cell]
    return dict(kind=kind, ds=ds, buf=buf, live=live, saved=[t.clone() for t in live],
                steps=case["steps"])


def _state_out(buf, cell):
    return dict({k: buf[k] for k in ("pos", "vel", "m_w", "m_s", "xi", "T_p", "grid", "mat", "dml",
                                     "water", "no_cols")}, cell=cell)


def run(state):
    s = state
    if s["kind"] == "step":
        ds = s["ds"]
        torch._foreach_copy_(s["live"], s["saved"])   # back to the checkpoint
        ds.prepare()
        ds.adv_step(s["steps"], graph=True)
        return _state_out(s["buf"], ds.cell)
    if s["kind"] == "batch":
        s["batch"].adv_step(1, graph=True)
        return _state_out(s["buf"], torch.cat([m.cell for m in s["batch"].members]))
    if s["kind"] == "dropin":
        st = s["st"]
        integration.integrate_adv_step_np(*[st[k] for k in integration._STATE_KEYS],
                                          draws=s["draws"], seed=s["seed"],
                                          precision=s["precision"], col_step=s["col_step"])
        s["col_step"] += st["no_col_per_adv"]
        return {k: st[k] for k in ("pos", "vel", "cells", "rel_pos", "m_w", "m_s", "xi", "T_p",
                                   "water_removed", "grid_scalar_fields", "grid_mat_prop",
                                   "delta_m_l", "no_cols")}
    if s["kind"] == "box":
        no_cols = np.zeros(2, dtype=np.int64)
        sip = [s["xis"].copy(), s["masses"].copy()]
        if s["method"] is not None:
            sip += [s["radii"].copy(), s["vel"].copy(), s["rho"]]
        xs, ms, _ = collision.simulate_collisions(tuple(sip), s["kernel"], s["name"], s["method"],
                                                  1.0, 1.0, float(s["steps"]), float(s["steps"]),
                                                  no_cols, s["seed"], draws="philox")
        return dict(xis=xs, masses=ms, no_cols=no_cols, final=sip[:4])
    J = adjoint.objective(s["model"], s["m_s"], s["kappa"], s["flux"], weights=s["weights"],
                          checkpoint_every=10)
    g = torch.autograd.grad(J, [s["m_s"], s["kappa"], s["flux"]])
    return dict(J=J.detach(), grad_m_s=g[0], grad_kappa=g[1], grad_flux=g[2])


def work(case):
    kind = case["kind"]
    if kind == "box":
        # every pair's probability and uniform draw once per step; the SIPs in and out
        n = case["sips"]
        pairs = n * (n - 1) // 2
        return {"bytes": 64.0 * n, "flops": 10.0 * pairs * case["steps"]}
    C, M = case["nx"] * case["nz"], case.get("members", 1)
    n = C * case["spc"] * M
    cells = 8.0 * C * M * (2 * 17 + 8)
    if kind == "adjoint":
        # per sub-step forward and backward: the map (3 evaluations) and its derivatives; the
        # tape of masses and cells written and read once
        sub = 10 * case["steps"]
        return {"bytes": n * (2 * 12.0 * sub + 40.0) + cells, "flops": n * sub * (500.0 + 3000.0)}
    steps = case.get("steps", 1)
    # state in: pos, vel, m_w, m_s, xi, cell; out: pos, vel, m_w, xi, m_s, cell, T_p
    byt = n * (60.0 + 68.0) + cells
    if kind == "dropin":
        byt *= 2.0   # over the host link and through HBM
    return {"bytes": byt, "flops": n * steps * 10 * 600.0}


# ---------------------------------------------------------------------------
# the same results in 64 bits with plain torch and numpy
def _mass_rate(sol, m_w, m_s, a, ks, w_s, rho_p, R_p, sigma_p):
    T = a["T"]
    l_a = 1.0E-6 * (R_p + (C_ALPHA[0] + C_ALPHA[1] * (T - T_A0)) * a["K"] / a["p"])
    l_b = 1.0E-6 * (R_p + C_BETA[0] * (1.0 + C_BETA[1] * (T - T_A0)) * a["D_v"])
    inv = 1.0E18 / (m_w + m_s)
    act, sig = (ACT_AS, SIGMA_AS) if sol == "AS" else (ACT_NACL, SIGMA_NACL)
    if sol == "AS":
        drho = -a["rho_w"] * inv / rho_p * w_s * _poly(_deriv(RHO_AS), w_s)
    else:
        drho = -w_s * inv / rho_p * (RHO_NACL[1] + 2.0 * RHO_NACL[3] * w_s + RHO_NACL[4] * T)
    a_w = 1.0 + ks * (_poly(act, w_s) - 1.0)
    da_w = -ks * inv * w_s * _poly(_deriv(act), w_s)
    dsig = -sig * a["sig_w"] * inv * (w_s / ((1. - w_s) * (1. - w_s)))
    dRR = (inv - drho) / 3.0
    dR = 1.0E-6 * dRR * R_p
    eps = 2.0E6 * sigma_p / (R_V * T * rho_p * R_p)
    kel = torch.exp(eps)
    S_eq = a_w * kel
    dS = da_w * kel + S_eq * eps * (dsig / sigma_p - drho - dRR)
    c1 = a["L_v"] ** 2 / (R_V * a["K"] * T * T)
    c2 = R_V * T / (a["D_v"] * a["e_s"])
    f3 = 1.0 / (l_a * S_eq * c1 + l_b * c2)
    f1f3 = 4.0 * math.pi * R_p * R_p * f3
    dg1 = (dS * l_a + S_eq * dR) * c1 + dR * c2
    f2 = a["S"] - S_eq
    return 1.0E6 * f1f3 * f2, 1.0E-12 * f1f3 * (f2 * (2.0 * dRR - f3 * dg1) - dS)


def _radius(m, rho):
    return (m / (FOUR_THIRDS_PI * rho)) ** (1.0 / 3.0)


def _newton(sol, m_w, m_s, a, ks, dt, no_iter):
    def damp(x):
        ok = x < 0.9
        return torch.where(ok, 1.0 / (1.0 - torch.where(ok, x, torch.zeros_like(x))),
                           torch.full_like(x, 10.0))
    floor = m_s * (W_MAX_INV - 1.0)
    w = m_s / (m_w + m_s)
    if sol == "AS":
        rho = a["rho_w"] * _poly(RHO_AS, w)
    else:
        T = a["T"]
        rho = (RHO_NACL[0] + RHO_NACL[1] * w + RHO_NACL[2] * T + RHO_NACL[3] * w * w
               + RHO_NACL[4] * w * T + RHO_NACL[5] * T * T)
    sig = a["sig_w"] * (1.0 + (SIGMA_AS if sol == "AS" else SIGMA_NACL) * w / (1. - w))
    g, dg = _mass_rate(sol, m_w, m_s, a, ks, w, rho, _radius(m_w + m_s, rho), sig)
    m = torch.maximum(floor, m_w + dt * g * damp(dt * dg))
    for _ in range(no_iter - 1):
        w = m_s / (m + m_s)
        rho = a["rho_w"] * _poly(RHO_AS, w)
        sig = a["sig_w"] * (1.0 + SIGMA_AS * w / (1. - w))
        g, dg = _mass_rate(sol, m, m_s, a, ks, w, rho, _radius(m + m_s, rho), sig)
        m = torch.maximum(floor, m + (dt * g + m_w - m) * damp(dt * dg))
    return m


def _limiter(a0, a1, a2):
    big = (a1 - a2).abs() > 1.0E-8 * (a0 - a1).abs()
    r = torch.where(big, (a0 - a1) / torch.where(big, a1 - a2, torch.ones_like(a1)),
                    (a0 - a1) * 1.0E8 * torch.sign(a1 - a2))
    return torch.clamp_min(torch.minimum(2.0 * r, torch.clamp_max((1.0 + 2.0 * r) / 3.0, 2.0)), 0.0)


def _faces(f, u, n):
    a0, a1, a2, an = f[2:n + 3], f[1:n + 2], f[0:n + 1], f[3:n + 4]
    return torch.where(u >= 0.0, u * (a1 + 0.5 * _limiter(a0, a1, a2) * (a1 - a2)),
                       u * (a0 + 0.5 * _limiter(a1, a0, an) * (a0 - an)))


def _increment(f, prof, st, flux, rdi, dt):
    nx, nz = f.shape
    dx, dz = (float(v) for v in st["grid_steps"])
    F = _faces(torch.cat([f[nx - 2:], f, f[:2]], 0), flux[0][:, :nz], nx)
    t = f.t()
    G = _faces(torch.cat([t[:1], t[:1], t, t[-1:], t[-1:]], 0), flux[1][:nx, :].t(), nz)
    G = torch.cat([torch.zeros_like(G[:1]), G[1:-1], torch.zeros_like(G[:1])], 0)
    inc = -dt * ((F[1:] - F[:-1]) / dx + ((G[1:] - G[:-1]) / dz).t()) * rdi
    if st["act_relaxation"]:
        dev = f.device
        trel = torch.as_tensor(st["relaxation_time_profile"], device=dev)
        inc = inc + dt * (torch.as_tensor(prof, device=dev) - f.sum(0) / nx) / trel
    return inc


def _wind(gv, i, j, a, b, nz):
    nx1, nz1 = gv.shape[1], gv.shape[2]
    at = lambda q, ii, jj: gv[q, torch.remainder(ii, nx1), torch.remainder(jj, nz1)]  # noqa: E731

    def bilin(q, ii, jj, p, s):
        return (p * (s * at(q, ii + 1, jj + 1) + (1 - s) * at(q, ii + 1, jj))
                + (1 - p) * (s * at(q, ii, jj + 1) + (1 - s) * at(q, ii, jj)))
    edge = ((j == 0) & (b <= 0.5)) | ((j == nz - 1) & (b >= 0.5))
    up = (b > 0.5).to(j.dtype)
    u = torch.where(edge, a * at(0, i + 1, j) + (1 - a) * at(0, i, j),
                    bilin(0, i, j - 1 + up, a, b + 0.5 - up))
    rt = (a > 0.5).to(j.dtype)
    return u, bilin(1, i - 1 + rt, j, a + 0.5 - rt, b)


class _Exact:
    """Advection steps without collisions in torch, FP64."""

    def __init__(self, st, m_s, kappa, flux_scale, sol):
        t = lambda x: torch.as_tensor(x, dtype=F64, device="cuda").clone()  # noqa: E731
        self.st, self.sol, self.ks = st, sol, kappa / 0.6
        self.nx, self.nz = (int(v) for v in st["grid_no_cells"])
        self.dx, self.dz = (float(v) for v in st["grid_steps"])
        self.V, self.dt = float(st["grid_volume_cell"]), float(st["dt_sub"])
        g = t(st["grid_scalar_fields"])
        self.gsf0, self.Th, self.rv, self.rho_d = g, g[2], g[4], g[3]
        self.x, self.z = t(st["pos"])
        self.u, self.w = t(st["vel"])
        self.m_w, self.m_s, self.xi = t(st["m_w"]), m_s, t(st["xi"])
        c = torch.as_tensor(st["cells"], device="cuda")
        self.i, self.j = c[0].clone(), c[1].clone()
        self.act = torch.ones_like(self.i, dtype=torch.bool)
        self.gv, self.flux = t(st["grid_velocity"]), t(st["grid_mass_flux_air_dry"]) * flux_scale
        self.water = torch.zeros(1, dtype=F64, device="cuda")
        self.T_p = t(st["T_p"])
        self.dml = torch.zeros(self.nx, self.nz, dtype=F64, device="cuda")

    def move(self, dt):
        x_max, z_cap = self.nx * self.dx, self.nz * self.dz * 0.999999
        self.x = torch.remainder(self.x + dt * self.u, x_max)
        self.z = torch.clamp_max(self.z + dt * self.w, z_cap)
        down = self.act & (self.z <= 0.0)
        if bool(down.any()):
            self.water = self.water + (self.xi * self.m_w.detach())[down].sum()
            self.z = torch.where(down, -0.01 * self.dz, self.z)
            self.u = torch.where(down, 0.0, self.u)
            self.w = torch.where(down, 0.0, self.w)
            self.act = self.act & ~down
        self.i = torch.where(self.act, (self.x / self.dx).floor().long(), self.i)
        self.j = torch.where(self.act, (self.z / self.dz).floor().long(), -1)

    def sub_step(self, dt_pos, dTh, drv):
        dt, c = self.dt, self.i * self.nz + self.j.clamp(min=0)
        a = _ambient(self.Th, self.rv, self.rho_d)
        at = {k: v.reshape(-1)[c] for k, v in a.items()}
        self.T_p = at["T"].detach()
        m = torch.where(self.act, _newton(self.sol, self.m_w, self.m_s, at, self.ks, dt,
                                          int(self.st["no_iter_impl_mass"])), self.m_w)
        dm = torch.where(self.act, (m - self.m_w) * self.xi, torch.zeros_like(m))
        dml = torch.zeros(self.nx * self.nz, dtype=F64, device="cuda").index_add(0, c, dm)
        dml = dml.reshape(self.nx, self.nz) * 1.0E-18
        self.m_w, self.dml = m, dml
        with torch.no_grad():   # drag and motion
            mp = m + self.m_s
            rho = at["rho_w"] * _poly(RHO_AS, self.m_s / mp)
            R = _radius(mp, rho)
            uf, wf = _wind(self.gv, self.i, self.j, self.x / self.dx - self.i,
                           self.z / self.dz - self.j, self.nz)
            dev = torch.sqrt((uf - self.u) ** 2 + (wf - self.w) ** 2)
            Re = 2.0E-6 * at["rho_f"] * R * dev / at["mu"]
            k = 4.5E12 * dt * at["mu"] / (rho * R * R)
            k = torch.where(Re > 0.5, k * torch.where(Re < 1000.0, 1 + 0.15 * Re ** 0.687,
                                                      0.0183333333333 * Re), k)
            self.u = torch.where(self.act, (self.u + k * uf) / (1.0 + k), self.u)
            self.w = torch.where(self.act, (self.w + k * wf - dt * float(self.st["g_set"]))
                                 / (1.0 + k), self.w)
            self.move(dt_pos)
        mdi = self.gsf0[8]
        Th, rv = self.Th + dTh, self.rv + drv - dml * mdi
        ToT = (R_D / 1.0E5 * self.rho_d * Th) ** KF2
        self.Th = Th + ToT * (a["L_v"] * dml) / (C_PD * self.rho_d * self.V * (1.0 + rv * HEAT_RV))
        self.rv = rv

    def adv_step(self):
        st, dt, rdi, S = self.st, self.dt, self.gsf0[9], int(self.st["scale_dt_cond"])
        with torch.no_grad():
            self.move(0.5 * dt)
        inc = lambda: (_increment(self.Th, st["init_profile_Theta"], st, self.flux, rdi, dt),  # noqa: E731
                       _increment(self.rv, st["init_profile_r_v"], st, self.flux, rdi, dt))
        d1 = inc()
        for _ in range(S):
            self.sub_step(dt, *d1)
        d2 = inc()
        d2 = 2.0 * d2[0] - d1[0], 2.0 * d2[1] - d1[1]
        for k in range(S):
            self.sub_step(dt if k < S - 1 else 0.5 * dt, *d2)

    def fields(self):
        a = _ambient(self.Th, self.rv, self.rho_d)
        g = self.gsf0
        gsf = torch.stack([a["T"], a["p"], self.Th, self.rho_d, self.rv, g[5], a["S"], a["e_s"],
                           g[8], g[9]])
        gmp = torch.stack([a["K"], a["D_v"], a["L_v"], a["sig_w"], C_PD * (1 + 0.897 * self.rv),
                           a["mu"], a["rho_f"]])
        return gsf, gmp


def _uniforms(seed, step, n, i, dev="cuda"):
    """Philox4x32-10 uniforms of the pairs (i, j), j > i, of n SIPs."""
    k = i * n - i * (i + 1) // 2 + torch.arange(n - i - 1, device=dev, dtype=torch.int64)
    M32 = 0xffffffff
    c = k >> 1
    x0, x1 = c & M32, c >> 32
    x2, x3 = torch.full_like(c, step & M32), torch.full_like(c, step >> 32)
    k0, k1 = seed & M32, seed >> 32
    for _ in range(10):
        p0, p1 = x0 * 0xD2511F53, x2 * 0xCD9E8D57
        x0, x1, x2, x3 = (((p1 >> 32) & M32) ^ x1 ^ k0, p1 & M32,
                          ((p0 >> 32) & M32) ^ x3 ^ k1, p0 & M32)
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    odd = (k & 1) != 0
    hi, lo = torch.where(odd, x2, x0), torch.where(odd, x3, x1)
    return ((hi >> 5) * 67108864 + (lo >> 6)).to(F64).cpu().numpy() / 9007199254740992.0


def _beard(R):
    rho_w, rho_a, mu, sigma, gr, l0 = 1.0E3, 1.225, 1.818E-5, 73.0E-3, 9.80665, 6.62E-2
    d = rho_w - rho_a
    v1 = d * gr / (4.5 * mu) * (1.0 + 1.257 * l0 / R) * R * R * 1.0E-12
    Y = np.log(32.0E-18 * R ** 3 * rho_a * d * gr / (3.0 * mu * mu))
    v2 = (mu * (1.0 + 1.257 * l0 / R) / (rho_a * R * 2.0E-6)
          * np.exp(_poly((-0.327815e-5, 0.855176e-4, -0.578878e-3, -0.987059e-3, -0.153193e-2,
                          0.992696, -0.318657e1), Y)))
    NP = (sigma ** 3 * rho_a * rho_a / (mu ** 4 * d * gr)) ** (1.0 / 6.0)
    Y = np.log(16.0E-12 * R * R * d * gr / (3.0 * sigma) * NP)
    v3 = (mu * NP / (rho_a * R * 2.0E-6)
          * np.exp(_poly((0.238449e-2, -0.542819e-1, 0.475294, -0.204914e1, 0.523778e1,
                          -0.500015e1), Y)))
    return np.where(R < 10.0, v1, np.where(R < 535.0, v2, np.where(R < 3500.0, v3, 9.04929248)))


def _box_exact(case, seed):
    """The box model row by row: the pairs of a row are looked at together, and
    again after each collection from the pair behind it on."""
    X, Ms, R = (v.copy() for v in _box(case, seed))
    n, tab, v = X.size, None, None
    x0, m0 = X.copy(), Ms.copy()
    cols = 0
    if case["method"] != "golovin":
        b = _base(dict(nx=8, nz=8, kernel=case["method"]), 1)
        E, nb, lo, bl = (b[k] for k in ("E_col_grid", "no_kernel_bins", "R_kernel_low_log",
                                        "bin_factor_R_log"))
        tab = lambda r: np.clip(((np.log(r) - lo) / bl + 0.5).astype(np.int64), 0, nb - 1)  # noqa: E731
        v = _beard(R)
    for step in range(case["steps"]):
        K = tab(R) if tab else None
        for i in range(n - 1):
            r, j0 = _uniforms(seed, step, n, i), i + 1
            while j0 < n:
                xm = np.maximum(X[i], X[j0:])
                if tab is None:
                    p = xm * ((Ms[i] + Ms[j0:]) * 1.5E-18)
                else:
                    Rs = R[i] + R[j0:]
                    p = xm * (math.pi * Rs * Rs * E[K[i], K[j0:]] * np.abs(v[i] - v[j0:]) * 1.0E-12)
                hit = np.flatnonzero((p > 1.0) | (p > r[j0 - i - 1:]))
                if not hit.size:
                    break
                j = j0 + int(hit[0])
                pc = float(p[hit[0]])
                cols += 1
                if cols > 20000:
                    return None   # a row at a time would take too long
                a, b2 = (i, j) if X[i] <= X[j] else (j, i)
                if pc > 1.0:
                    Ms[a] += pc * Ms[b2]
                    X[b2] -= pc * X[a]
                    new = (a,)
                elif (X[b2] - X[a]) / X[b2] < 1.0E-5:
                    s = X[a] + X[b2]
                    Ms[a] = Ms[b2] = 2.0 * (X[a] * Ms[a] + X[b2] * Ms[b2]) / s
                    X[b2] = 0.35 * s
                    X[a] = 0.5 * s - X[b2]
                    new = (a, b2)
                else:
                    Ms[a] += Ms[b2]
                    X[b2] -= X[a]
                    new = (a,)
                if tab is not None:
                    for q in new:
                        R[q] = (Ms[q] / (FOUR_THIRDS_PI * 1000.0)) ** (1.0 / 3.0)
                        K[q] = tab(R[q:q + 1])[0]
                j0 = j + 1
        if tab is not None:
            v = _beard(R)
    out = dict(xis=np.stack([x0, X]), masses=np.stack([m0, Ms]), no_cols=None, final=[X, Ms])
    if tab is not None:
        out["final"] += [R, v]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "box":
        return _box_exact(case, seed) if case["sips"] <= 1200 or case["method"] == "golovin" else None
    if kind == "adjoint" and not case["collisions"]:
        st = _members(case, seed, 1)[0][0]
        m_s = st["m_s"].clone().requires_grad_()
        kappa = torch.tensor(0.6, dtype=F64, device="cuda", requires_grad=True)
        flux = torch.tensor(1.0, dtype=F64, device="cuda", requires_grad=True)
        e = _Exact(st, m_s, kappa, flux, "AS")
        for _ in range(case["steps"]):
            e.adv_step()
        width = e.nx * e.dx
        w = e.xi * 1.0E-18 / width
        w = torch.where(e.act, w, 100.0 * w / (case["steps"] * float(st["dt"])))
        J = (w * e.m_w).sum()
        g = torch.autograd.grad(J, [m_s, kappa, flux])
        return dict(J=J.detach(), grad_m_s=g[0], grad_kappa=g[1], grad_flux=g[2])
    if kind == "step" and not case["collisions"]:
        sts, buf = _members(case, seed, 1)
        with torch.no_grad():
            e = _Exact(sts[0], sts[0]["m_s"].clone(), 0.6, 1.0, case["solute"])
            for _ in range(case["steps"]):
                e.adv_step()
            n = e.m_w.numel()
            gsf, gmp = e.fields()
            full = lambda k, *v: torch.cat([*v, buf[k][len(v) * n:]])  # noqa: E731
            return dict(pos=full("pos", e.x, e.z), vel=full("vel", e.u, e.w),
                        m_w=full("m_w", e.m_w), m_s=buf["m_s"], xi=buf["xi"],
                        T_p=full("T_p", e.T_p), grid=gsf.reshape(1, 10, -1),
                        mat=gmp.reshape(1, 7, -1), dml=e.dml.reshape(1, -1), water=None,
                        no_cols=None, cell=None)
    return None
