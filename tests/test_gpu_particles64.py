"""The FP64 particle sub-step outside its common path: the sizes and steps that
leave its two-float arithmetic, cell and domain edges, SIPs removed together, sums
beyond the integer range, against the oracle's sub-step; and the reverse of the
condensation map for the evaluation counts at its limits.

Tolerances: 1e-10 is the product's stated agreement.  The masses are compared
with the same map in long double: in these steps (SIPs far from equilibrium) FP64
itself, the oracle's too, loses up to 1e-10 to the residual S - S_eq, a difference
of numbers near 1 that the later evaluations amplify.  A velocity is
one rounding of a sum of terms no larger than 20 m/s: 1e-10 relative, 1e-12 m/s
absolute.  Removed water is a sum of positive terms: 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(sol, n=4000, seed=2):
    from lacmopy_gb300 import synthetic
    rng = np.random.default_rng(seed)
    st = synthetic.make_icmw_state(Nx=7, Nz=5, no_spcm=(1, 1), seed=4, r_tot=12.5E-3)
    nx, nz = 7, 5
    dx, dz = st["grid_steps"]
    i, j = rng.integers(0, nx, n), rng.integers(0, nz, n)
    fx, fz = rng.random(n), rng.random(n)
    edge = rng.random(n) < 0.3
    pick = np.array([1e-13, 1e-9, 1e-5, 0.25, 0.5, 0.5 + 1e-15, 1 - 1e-5, 1 - 1e-9])
    fx[edge] = rng.choice(pick, edge.sum())
    fz[edge] = rng.choice(pick, edge.sum())
    j[:300] = 0                       # near the ground, falling
    fz[:300] = 1e-3 * rng.random(300)
    pos = np.array([(i + fx) * dx, (j + fz) * dz])
    i, j = np.floor(pos[0] / dx).astype(int), np.floor(pos[1] / dz).astype(int)
    # dry radii 2 nm to 1 um, wet radii from a little above to 2 mm
    R_s = np.exp(rng.uniform(np.log(2e-3), 0.0, n))
    m_s = 4.18879 * 1774.0 * R_s ** 3
    R_w = np.maximum(R_s * 1.02, np.exp(rng.uniform(np.log(3e-3), np.log(2e3), n)))
    m_w = np.maximum(4.18879e3 * R_w ** 3 - m_s * 0.5, m_s * 0.3)
    m_s[-6:-3] = 1e-24                # below the two-float range
    m_w[-6:-3] = (1e-23, 1e-20, 1e-2)
    m_w[-3:] = 1e31                   # above it
    vel = rng.normal(0.0, 1.0, (2, n))
    vel[1] -= np.minimum(8e-3 * R_w, 9.0)
    vel[1, :300] = -2.0
    st.update(pos=pos, vel=vel, cells=np.array([i, j], dtype=np.int64),
              rel_pos=np.array([pos[0] / dx - i, pos[1] / dz - j]), m_w=m_w, m_s=m_s,
              xi=np.exp(rng.uniform(0.0, 20.0, n)), T_p=np.ones(n),
              active_ids=np.full(n, True), id_list=np.arange(n), solute_type=sol)
    return st


def _poly(par, x):
    r = float(par[0]) * x + float(par[1])
    for a in par[2:]:
        r = r * x + float(a)
    return r


def _newton_long(st, no_iter, dt=0.1):
    """integration.py:728-836 with the mass rate of microphysics.py:1239-1469
    in long double, for the active SIPs of ``st``."""
    from lacmopy_gb300 import constants as c
    L = np.longdouble
    act = st["active_ids"] & (np.arange(st["m_w"].size) < st["m_w"].size - 6)
    i, j = st["cells"][:, act]
    f = [L(v[i, j]) for v in st["grid_scalar_fields"]]
    g = [L(v[i, j]) for v in st["grid_mat_prop"]]
    T, p, S, es, K, Dv, Lv = f[0], f[1], f[6], f[7], g[0], g[1], g[2]
    mw, ms = L(st["m_w"][act]), L(st["m_s"][act])
    tau = 1 - T / L(647.096)
    sigw = L(0.2358) * tau ** L(1.256) * (1 - L(0.625) * tau)
    pw = [float(v) for v in c.par_water_dens]
    rhow = pw[0] + pw[1] * (T - pw[2]) ** 2
    la = (c.c_alpha_1 + c.c_alpha_2 * (T - 289)) * K / p
    lb = c.c_beta_1 * (1 + c.c_beta_2 * (T - 289)) * Dv
    Rv = c.specific_gas_constant_water_vapor
    c1, c2 = Lv * Lv / (Rv * K * T * T), Rv * T / (Dv * es)
    AS = st["solute_type"] == "AS"
    q = [float(v) for v in c.par_sol_dens_NaCl]
    s1 = c.par_sigma_AS if AS else c.par_sigma_NaCl

    def rate(m, w, rho, sig):
        R = (c.four_pi_over_three_inv * (m + ms) / rho) ** (L(1) / 3)
        inv = L(1e18) / (m + ms)
        if AS:
            dr = -rhow * inv / rho * w * _poly(c.par_rho_deriv_AS, w)
            aw, da = _poly(c.par_wat_act_AS, w), -inv * w * _poly(c.par_wat_act_deriv_AS, w)
        else:
            dr = -w * inv / rho * (q[1] + 2 * q[3] * w + q[4] * T)
            aw, da = _poly(c.par_wat_act_NaCl, w), -inv * w * _poly(c.par_wat_act_deriv_NaCl, w)
        ds = -s1 * sigw * inv * (w / (1 - w) ** 2)
        dRR = (inv - dr) / 3
        dR = L(1e-6) * dRR * R
        eps = L(2e6) * sig / (Rv * T * rho * R)
        Se = aw * np.exp(eps)
        dS = da * np.exp(eps) + Se * eps * (ds / sig - dr - dRR)
        A, B = L(1e-6) * (R + la), L(1e-6) * (R + lb)
        f3 = 1 / (A * Se * c1 + B * c2)
        f1 = 4 * L(np.pi) * R * R * f3
        dg = (dS * A + Se * dR) * c1 + dR * c2
        return L(1e6) * f1 * (S - Se), L(1e-12) * f1 * ((S - Se) * (2 * dRR - f3 * dg) - dS)

    def damp(x):
        return np.where(x < L(0.9), 1 / (1 - np.where(x < L(0.9), x, 0)), L(10))
    floor = ms * (c.w_s_max_AS_inv - 1)
    w = ms / (mw + ms)
    rho = (rhow * _poly(c.par_rho_AS, w) if AS else
           q[0] + q[1] * w + q[2] * T + q[3] * w * w + q[4] * w * T + q[5] * T * T)
    G, dG = rate(mw, w, rho, sigw * (1 + s1 * w / (1 - w)))
    m = np.maximum(floor, mw + L(dt) * G * damp(L(dt) * dG))
    for _ in range(no_iter - 1):
        w = ms / (m + ms)
        G, dG = rate(m, w, rhow * _poly(c.par_rho_AS, w),
                     sigw * (1 + c.par_sigma_AS * w / (1 - w)))
        m = np.maximum(floor, m + (L(dt) * G + mw - m) * damp(L(dt) * dG))
    # drag (integration.py:699-718) in the interpolated wind (grid.py:257-323)
    w = ms / (m + ms)
    rho = rhow * _poly(c.par_rho_AS, w)
    R = (c.four_pi_over_three_inv * (m + ms) / rho) ** (L(1) / 3)
    gv, (dx, dz) = L(st["grid_velocity"]), st["grid_steps"]
    nz = int(st["grid_no_cells"][1])
    a, b = L(st["pos"][0, act]) / dx - i, L(st["pos"][1, act]) / dz - j

    def at(k, ii, jj):
        return gv[k, ii % gv.shape[1], jj % gv.shape[2]]

    def bil(k, ii, jj, x, y):
        return (x * (y * at(k, ii + 1, jj + 1) + (1 - y) * at(k, ii + 1, jj))
                + (1 - x) * (y * at(k, ii, jj + 1) + (1 - y) * at(k, ii, jj)))
    up, rt = (b > 0.5).astype(int), (a > 0.5).astype(int)
    edge = ((j == 0) & (b <= 0.5)) | ((j == nz - 1) & (b >= 0.5))
    uf = np.where(edge, a * at(0, i + 1, j) + (1 - a) * at(0, i, j),
                  bil(0, i, j - 1 + up, a, b + L(0.5) - up))
    wf = bil(1, i - 1 + rt, j, a + L(0.5) - rt, b)
    u, v = L(st["vel"][:, act])
    Re = L(2e-6) * g[6] * R * np.sqrt((uf - u) ** 2 + (wf - v) ** 2) / g[5]
    k = L(4.5e12) * L(dt) * g[5] / (rho * R * R)
    k = np.where(Re > 0.5, k * np.where(Re < 1000, 1 + L(0.15) * Re ** L(0.687),
                                        L(0.0183333333333) * Re), k)
    out, vel = L(st["m_w"]), L(st["vel"])
    out[act] = m
    vel[:, act] = (u + k * uf) / (1 + k), (v + k * wf - L(dt) * L(9.80665)) / (1 + k)
    return out, vel


def _sub_step(mod, st, no_iter, dt_pos):
    mod.propagate_particles_subloop_step_np(
        st["grid_scalar_fields"], st["grid_mat_prop"], st["grid_velocity"], st["grid_no_cells"],
        st["grid_ranges"], st["grid_steps"], st["pos"], st["vel"], st["cells"], st["rel_pos"],
        st["m_w"], st["m_s"], st["xi"], st["water_removed"], None, st["active_ids"], st["T_p"],
        st["solute_type"], st["delta_m_l"], 0.1, dt_pos, no_iter, 9.80665)


@pytest.mark.parametrize("sol", ["AS", "NaCl"])
@pytest.mark.parametrize("no_iter,n", [(3, 4000), (1, 700), (5, 129)])
def test_sub_step_vs_oracle(oracle_nb, sol, no_iter, n):
    from lacmopy_gb300 import integration as I
    a = _state(sol, n=max(n, 400))
    b = {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in a.items()}
    for dt_pos in (0.1, 0.05):   # the second sub-step meets removed SIPs
        m, vel = _newton_long(a, no_iter)
        _sub_step(I, a, no_iter, dt_pos)
        _sub_step(oracle_nb, b, no_iter, dt_pos)
        assert (~b["active_ids"]).sum() >= 50
        assert np.array_equal(a["cells"], b["cells"])
        assert np.array_equal(a["active_ids"], b["active_ids"])
        assert float(np.abs(a["m_w"] / m - 1)[:-6].max()) <= 1e-10
        # out of any range (exp overflows): the oracle's values, NaN among them
        np.testing.assert_allclose(a["m_w"][-6:], b["m_w"][-6:], rtol=1e-10)
        vel[:, ~b["active_ids"]] = 0.0   # removed at the ground
        assert (np.abs(a["vel"] - vel) <= 1e-10 * np.abs(vel) + 1e-12)[:, :-6].all()
        np.testing.assert_allclose(a["vel"][:, -6:], b["vel"][:, -6:], rtol=1e-10, atol=1e-12)
        np.testing.assert_allclose(a["pos"], b["pos"], rtol=1e-12, atol=1e-12)
        np.testing.assert_allclose(a["rel_pos"], b["rel_pos"], rtol=1e-9, atol=1e-11)
        np.testing.assert_allclose(a["water_removed"], b["water_removed"], rtol=1e-12)
        assert np.array_equal(a["T_p"], b["T_p"])


def test_sums_beyond_the_integer_range(oracle_nb):
    """A product dm xi of 2^60 fg and more, and one NaN: the plain FP64 sum."""
    from lacmopy_gb300 import integration as I
    a = _state("AS", n=500)
    a["xi"][310] = 1e40
    a["m_w"][320] = np.nan
    b = {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in a.items()}
    _sub_step(I, a, 3, 0.1)
    _sub_step(oracle_nb, b, 3, 0.1)
    assert np.isnan(b["delta_m_l"]).any() and np.nanmax(np.abs(b["delta_m_l"])) > 1e10
    np.testing.assert_allclose(a["delta_m_l"], b["delta_m_l"], rtol=1e-8,
                               atol=1e-12 * np.nanmedian(np.abs(b["delta_m_l"])))


@pytest.mark.parametrize("no_iter", [1, 2, 8, 9])
def test_map_gradient_vs_torch(no_iter):
    """Evaluation counts up to and beyond the reverse's stored masses (8),
    against autograd through the FP64 restatement: the two-float partials are
    within 2^-42, 20 sub-steps deep."""
    import torch
    import torch_step_model as ref
    from lacmopy_gb300 import adjoint, synthetic
    st = synthetic.make_icmw_state(Nx=4, Nz=6, no_spcm=(3, 4), seed=6, kernel_type="Long_Bott",
                                   drizzle_fraction=0.3, r_tot=12.5E-3)
    model = adjoint.StepModel(st, 2)
    w = torch.rand(model.n, generator=torch.Generator().manual_seed(4), dtype=torch.float64)
    m_s = model.m_s0.clone().requires_grad_(True)
    kappa = torch.tensor(0.55, dtype=torch.float64, device="cuda", requires_grad=True)
    s = torch.tensor(1.1, dtype=torch.float64, device="cuda", requires_grad=True)
    J = adjoint.objective(model, m_s, kappa, s, weights=w.cuda(), no_iter=no_iter)
    g = torch.autograd.grad(J, [m_s, kappa, s])
    m_r = torch.as_tensor(st["m_s"], dtype=torch.float64).clone().requires_grad_(True)
    k_r = torch.tensor(0.55, dtype=torch.float64, requires_grad=True)
    s_r = torch.tensor(1.1, dtype=torch.float64, requires_grad=True)
    J_r = (w * ref.run(st, model.cells.cpu(), m_r, k_r, s_r, 2, no_iter,
                       events=ref.decode_events(model.events))).sum()
    r = torch.autograd.grad(J_r, [m_r, k_r, s_r])
    assert abs(float(J.detach()) - float(J_r.detach())) <= 1e-11 * abs(float(J_r.detach()))
    for x, y in zip(g, r):
        assert float((x.cpu() - y).abs().max()) <= 1e-9 * float(y.abs().max())


@pytest.mark.parametrize("solute", ["AS", "NaCl"])
def test_full_and_sparse_grids_agree(solute):
    """The conversions without FP64 instructions (states of more SIPs than are
    resident) give the bits of the plain ones: a state too small for them, and
    the same state twice in a batch that is large enough."""
    import copy
    from lacmopy_gb300 import BatchState, DeviceState, synthetic
    st = synthetic.make_icmw_state(Nx=25, Nz=25, no_spcm=(32, 40), seed=8, kernel_type="Long_Bott",
                                   drizzle_fraction=0.05, r_tot=11E-3)
    st["solute_type"] = solute
    assert 39000 < st["xi"].size < 77000   # between two and four blocks of 128 an SM
    one = DeviceState(copy.deepcopy(st), draws="philox", seed=5)
    one.adv_step(2)
    two = BatchState([copy.deepcopy(st), copy.deepcopy(st)], [5, 5], precision="fp64",
                     draws="philox")
    two.adv_step(2)
    a = one.snapshot()
    for m in range(2):
        b = two.snapshot(m)
        for k in ("m_w", "vel", "pos", "xi", "grid_scalar_fields", "water_removed"):
            assert np.array_equal(a[k], b[k]), k


def test_forward_of_a_full_grid_replays_the_product():
    """More SIPs than are resident: the replay takes the conversions without FP64
    instructions and the queue, and still gives the product's masses."""
    import torch
    from lacmopy_gb300 import adjoint, synthetic
    st = synthetic.make_icmw_state(Nx=40, Nz=40, no_spcm=(26, 38), seed=9, kernel_type="Long_Bott",
                                   drizzle_fraction=0.05, r_tot=11E-3)
    assert st["xi"].size > 100000
    model = adjoint.StepModel(st, 1)
    m_w, m_s, xi, Th, rv = model.run(full=True)
    torch.testing.assert_close(m_w, model.product.m_w, rtol=1e-11, atol=1e-30)
    torch.testing.assert_close(Th, model.product.gsf[2].reshape(-1), rtol=1e-13, atol=0)
