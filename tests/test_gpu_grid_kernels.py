"""Edges of the per-cell kernels: the upwind divergence on grids of one to five
cells a side, where stencils wrap around or are clamped to one cell, and the
binning's scan and work order at whole and broken tiles of 1024 cells."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc", [(0, 1), (1, 0), (0, 0), (1, 1)])
@pytest.mark.parametrize("shape", [(1, 1), (1, 4), (4, 1), (2, 2), (2, 3), (3, 2), (5, 33)])
def test_divergence_of_small_grids(oracle_py, shape, bc):
    from lacmopy_gb300 import integration as I
    nx, nz = shape
    rng = np.random.default_rng(nx * 10 + nz)
    f = 1.0 + 0.3 * rng.standard_normal(shape)
    if nx > 1:
        f[1] = f[0]   # equal neighbours: the limiter's other branch
    flux = rng.standard_normal((2, nx + 1, nz + 1))
    flux[:, 0] = 0.0
    a = I.compute_divergence_upwind_np(f, flux, np.array(shape), np.array([20.0, 25.0]), bc)
    b = oracle_py.compute_divergence_upwind_np(f, flux, np.array(shape), np.array([20.0, 25.0]), bc)
    # two fluxes of some 10 flops each: within 32 roundings of the largest flux
    tol = 32 * 2.0 ** -53 * np.abs(flux).max() * 4 * np.abs(f).max() / 20.0
    assert np.abs(a - b).max() <= tol


@pytest.mark.parametrize("shape", [(1, 2), (32, 32), (41, 25), (31, 33), (64, 33)])
@pytest.mark.parametrize("uneven", [False, True])
def test_binning_of_whole_and_broken_tiles(oracle_cr, shape, uneven):
    """2, 1023, 1024, 1025 and 2112 cells, all of one size class or of many:
    every pair of every cell gets its own draw, as in the oracle."""
    from lacmopy_gb300 import DeviceState, synthetic
    nx, nz = shape
    C = nx * nz
    rng = np.random.default_rng(C)
    counts = rng.integers(0, 9, C) if uneven else np.full(C, 5)
    n = int(counts.sum())
    spc = max(4, -(-n // max(1, (nx if nx > 2 else 4) * (nz if nz > 2 else 4))) + 1)
    st = synthetic.make_icmw_state(Nx=max(nx, 4), Nz=max(nz, 4), no_spcm=(spc, spc), seed=3,
                                   kernel_type="Long_Bott", drizzle_fraction=0.3, r_tot=12.5E-3)
    assert st["xi"].size >= n
    cell = np.repeat(np.arange(C), counts)[rng.permutation(n)]
    sel = rng.permutation(st["xi"].size)[:n]
    T = np.full(shape, 285.0)
    xi, mw, ms = (st[k][sel].copy() for k in ("xi", "m_w", "m_s"))
    vel = np.ascontiguousarray(st["vel"][:, sel])
    cells = np.array([cell // nz, cell % nz], dtype=np.int64)
    args = (st["dt_col_over_dV"] * 300.0, st["E_col_grid"], st["no_kernel_bins"],
            st["R_kernel_low_log"], st["bin_factor_R_log"])
    from lacmopy_gb300 import collision
    a = [v.copy() for v in (xi, mw, ms)]
    na = np.zeros(2, np.int64)
    collision.collision_step_Ecol_grid_R_all_cells_2D_multicomp_np(
        *a, vel, T, cells, np.array(shape), *args, na, "AS", draws="philox", seed=23, col_step=0)
    nb, cs = np.zeros(2, np.int64), np.zeros(1, np.int64)
    b = [v.copy() for v in (xi, mw, ms)]
    oracle_cr.collision_step_all_cells_philox(*b, vel, T, cells, np.array(shape), *args, nb, "AS",
                                              23, cs)
    assert nb.sum() > 0 or n < 100
    assert np.array_equal(na, nb)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
