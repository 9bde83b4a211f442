"""The per-cell thermodynamics (exp, log, root and quotients of
csrc/lacmo_math64.cuh) through the grid sub-step, against long double over the
atmosphere's range and beyond.

Tolerances, from the roundings of each field (u = 2^-53): Theta and r_v a handful
of u; T and p the exponential of a rounded argument below 1, 8 u; e_s and S the
exponential of 5420 / T (15 to 35, half an ulp of it 16 u, and T's 8 u times
5420 / T): 300 u; the rest follow T and p within 16 u."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(75, 75), (1, 1), (33, 1), (3, 11)])
def test_grid_sub_step_vs_long_double(nx, nz):
    from lacmopy_gb300 import constants as c
    from lacmopy_gb300 import integration as I
    L = np.longdouble
    rng = np.random.default_rng(nx)
    sh = (nx, nz)
    Th0, rho = rng.uniform(180.0, 420.0, sh), rng.uniform(0.2, 1.5, sh)
    rv0, V, p_ref = 10.0 ** rng.uniform(-7, -1.3, sh), 400.0, 1.0e5
    mdi = 1.0 / (rho * V)
    gsf = np.zeros((10,) + sh)
    gsf[2], gsf[3], gsf[4], gsf[8], gsf[9] = Th0, rho, rv0, mdi, 1.0 / rho
    gmp = np.zeros((7,) + sh)
    Lv0 = rng.uniform(2.3e6, 2.7e6, sh)
    gmp[2] = Lv0
    dTh, drv = rng.normal(0, 1e-3, sh), rng.normal(0, 1e-3, sh) * rv0
    dml = rng.normal(0, 0.1, sh) * rv0 * rho * V
    I.propagate_grid_subloop_step_np(gsf, gmp, p_ref, 1.0 / p_ref, dTh, drv, dml, V)
    R_d, R_v, cp = (L(v) for v in (c.specific_gas_constant_air_dry,
                                   c.specific_gas_constant_water_vapor,
                                   c.specific_heat_capacity_air_dry_NTP))
    Th, rv = L(Th0) + dTh, L(rv0) + (L(drv) - L(dml) * mdi)
    pri = L(1.0 / p_ref)
    Th = Th + (pri * R_d * rho * Th) ** L(c.kappa_factor2) * (L(Lv0) * dml) / (
        cp * rho * V * (1 + rv * c.heat_factor_r_v))
    pdr = (rho * Th * R_d * pri) ** L(c.kappa_factor)
    T = Th * pdr ** L(c.kappa_air_dry)
    p = pdr * p_ref * (1 + rv / c.epsilon_gc)
    es = L(2.53E11) * np.exp(-5420 / T)
    tau = 1 - T / L(647.096)
    ref = [(gsf[2], Th, 8), (gsf[4], rv, 4), (gsf[0], T, 8), (gsf[1], p, 12), (gsf[7], es, 300),
           (gsf[6], rho * rv * T * R_v / es, 300),
           (gmp[1], L(4.01218E-5) * T ** L(1.94) / p, 24),
           (gmp[5], L(1.458E-6) * T ** L(1.5) / (T + L(110.4)), 16),
           (gmp[3], L(0.2358) * tau ** L(1.256) * (1 - L(0.625) * tau), 16),
           (gmp[6], rho * (1 + rv), 4)]
    for k, (got, want, u) in enumerate(ref):
        err = float(np.abs(got / want - 1).max())
        assert err <= u * 2.0 ** -53, (k, err / 2.0 ** -53)
