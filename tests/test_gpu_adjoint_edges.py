"""The adjoint at the edges: cells without vapour, no scratch memory.

Tolerances: the two-float partials of a sub-step are within 2^-42 (2.3e-13) of the
terms they add up, which here stay within a factor of 100 of the largest entry:
1e-9 of that entry, as for states inside the range."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
F64 = torch.float64


def _state(r_v, floored=False):
    """Cell (1, 2) holds vapour r_v only; no drizzle, SIPs away from cell edges."""
    import numpy as np
    from lacmopy_gb300 import constants, synthetic
    st = synthetic.make_icmw_state(Nx=4, Nz=6, no_spcm=(3, 4), seed=6, kernel_type="Long_Bott",
                                   r_tot=12.5E-3)
    gsf = st["grid_scalar_fields"]
    gsf[6, 1, 2] *= r_v / gsf[4, 1, 2]
    gsf[4, 1, 2] = r_v
    dx, dz = st["grid_steps"]
    rel = 0.2 + 0.6 * np.random.default_rng(2).random((2, st["xi"].size))
    st["rel_pos"][:] = rel
    st["pos"][0] = (st["cells"][0] + rel[0]) * dx
    st["pos"][1] = (st["cells"][1] + rel[1]) * dz
    here = (st["cells"][0] == 1) & (st["cells"][1] == 2)
    if floored:   # as dry as the solute allows
        st["m_w"][here] = st["m_s"][here] * (constants.w_s_max_AS_inv - 1.0)
    assert here.sum() >= 5
    return st


@pytest.mark.parametrize("r_v", [0.0, 1e-45, 1e-30])
def test_sub_step_of_a_dry_cell(r_v):
    """The adjoints of Theta and r_v before one sub-step, and of m_s."""
    import torch_step_model as ref
    from lacmopy_gb300 import adjoint
    from lacmopy_gb300 import constants as c
    st = _state(r_v)
    model = adjoint.StepModel(st, 1, collisions=False)
    n, C, dev = model.n, model.C, "cuda"
    gen = torch.Generator().manual_seed(4)
    w = torch.rand(n, generator=gen, dtype=F64)
    wT, wr = torch.rand(C, generator=gen, dtype=F64), torch.rand(C, generator=gen, dtype=F64)
    m_w, m_s, xi, Th, rv = model.initial_state()
    tape_m = torch.empty(2 * n, dtype=F64, device=dev)
    tape_c = torch.empty(2 * C, dtype=F64, device=dev)
    model._sub_steps(m_w, m_s, Th, rv, 0.6, model.cells[0], n, 1, None, 3, tape_m, tape_c)
    # scales that weigh the masses, Theta and r_v alike
    lam = [w.to(dev), (1e3 * wT).to(dev), (1e6 * wr).to(dev), torch.zeros(C, dtype=F64, device=dev)]
    g_ms, g_k = torch.zeros(n, dtype=F64, device=dev), torch.zeros(1, dtype=F64, device=dev)
    model._sub_steps_bwd(m_s, 0.6, model.cells[0], n, 1, None, 3, tape_m, tape_c, lam, g_ms, g_k,
                         None)
    cell = model.cells[0].cpu().long()
    gsf = torch.as_tensor(st["grid_scalar_fields"], dtype=F64)
    T0, r0 = (gsf[q].reshape(C).clone().requires_grad_(True) for q in (2, 4))
    s0 = torch.as_tensor(st["m_s"], dtype=F64).clone().requires_grad_(True)
    mw0 = torch.as_tensor(st["m_w"], dtype=F64)
    rho_d, mdi = gsf[3].reshape(C), gsf[8].reshape(C)
    p_ref, V = float(st["p_ref"]), float(st["grid_volume_cell"])
    a = ref.ambient(T0, r0, rho_d, p_ref)
    m1 = ref.newton(mw0, s0, 1.0, {k: v[cell] for k, v in a.items()}, float(st["dt_sub"]), 3)
    dml = torch.zeros(C, dtype=F64).index_add(
        0, cell, (m1 - mw0) * torch.as_tensor(st["xi"], dtype=F64)) * 1e-18
    r1 = r0 - dml * mdi
    ToT = (c.specific_gas_constant_air_dry / p_ref * rho_d * T0) ** c.kappa_factor2
    T1 = T0 + ToT * (a["L_v"] * dml) / (c.specific_heat_capacity_air_dry_NTP * rho_d * V
                                        * (1.0 + r1 * c.heat_factor_r_v))
    J = (w * m1).sum() + 1e3 * (wT * T1).sum() + 1e6 * (wr * r1).sum()
    want = torch.autograd.grad(J, [T0, r0, s0])
    for x, y in zip((lam[1], lam[2], g_ms), want):
        assert bool(torch.isfinite(y).all()) and bool((y != 0).any())
        assert float((x.cpu() - y).abs().max()) <= 1e-9 * float(y.abs().max())
    k = 1 * model.nz + 2   # the dry cell itself
    assert abs(float(lam[2][k].cpu() - want[1][k])) <= 1e-9 * abs(float(want[1][k]))


def test_gradient_with_a_cell_that_stays_dry():
    """Its SIPs cannot lose more water: r_v = 0 in every sub-step."""
    import torch_step_model as ref
    from lacmopy_gb300 import adjoint
    st = _state(0.0, floored=True)
    st["grid_mass_flux_air_dry"][:] = 0.0
    st["grid_velocity"][:] = 0.0
    st["vel"][:] = 0.0
    st["act_relaxation"] = False
    model = adjoint.StepModel(st, 1, collisions=False)
    w = torch.rand(model.n, generator=torch.Generator().manual_seed(4), dtype=F64)
    m_s = model.m_s0.clone().requires_grad_(True)
    kappa = torch.tensor(0.55, dtype=F64, device="cuda", requires_grad=True)
    J = adjoint.objective(model, m_s, kappa, 1.0, weights=w.cuda(), no_iter=3)
    g = torch.autograd.grad(J, [m_s, kappa])
    m_r = torch.as_tensor(st["m_s"], dtype=F64).clone().requires_grad_(True)
    k_r = torch.tensor(0.55, dtype=F64, requires_grad=True)
    r = torch.autograd.grad((w * ref.run(st, model.cells.cpu(), m_r, k_r, 1.0, 1, 3)).sum(),
                            [m_r, k_r])
    for x, y in zip(g, r):
        assert bool(torch.isfinite(y).all())
        assert float((x.cpu() - y).abs().max()) <= 1e-9 * float(y.abs().max())


def _without_scratch(tmp_path):
    """The adjoint's object file with a scratch allocator that has nothing."""
    import ctypes
    import os
    import subprocess
    from lacmopy_gb300 import _lib, build
    build.build()
    src = tmp_path / "no_scratch.cu"
    src.write_text('#include "lacmo_internal.cuh"\nnamespace lacmo {\nvoid note_launches(int) {}\n'
                   'void* Scratch::get(size_t) { return nullptr; }\n}\n')
    out = str(tmp_path / "no_scratch.so")
    adj = os.path.join(build.BUILD, "k_adjoint.o")
    flags = build.ARCH + ["-std=c++17", "-I" + build.CSRC, "-Xcompiler", "-fPIC"]
    subprocess.run([build._nvcc(), "-shared", "-o", out, str(src), adj] + flags, check=True)
    lib = ctypes.CDLL(out)
    full = _lib.load()

    class Lib:
        def __getattr__(self, name):
            f = getattr(full, name)
            if name in ("lacmo_adj_forward", "lacmo_adj_backward"):
                g = getattr(lib, name)
                g.restype, g.argtypes = f.restype, f.argtypes
                return g
            return f
    return Lib()


@pytest.mark.parametrize("no_iter", [0, 3])
def test_gradient_without_scratch(tmp_path, no_iter):
    """Masses within 1e-11 (the FP64 map against the two-float one), gradients as
    above."""
    from lacmopy_gb300 import adjoint
    model = adjoint.StepModel(_state(5e-3), 1)
    w = torch.rand(model.n, generator=torch.Generator().manual_seed(4), dtype=F64).cuda()
    out = []
    for lib in (model.lib, _without_scratch(tmp_path)):
        model.lib = lib
        m_s = model.m_s0.clone().requires_grad_(True)
        kappa = torch.tensor(0.55, dtype=F64, device="cuda", requires_grad=True)
        s = torch.tensor(1.1, dtype=F64, device="cuda", requires_grad=True)
        J = adjoint.objective(model, m_s, kappa, s, weights=w, no_iter=no_iter)
        out.append((model.run(no_iter=no_iter)[0], *torch.autograd.grad(J, [m_s, kappa, s])))
    torch.testing.assert_close(out[1][0], out[0][0], rtol=1e-11, atol=0)
    for x, y in zip(out[1][1:], out[0][1:]):
        assert float((x - y).abs().max()) <= 1e-9 * float(y.abs().max())
