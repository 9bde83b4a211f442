"""The per-pair collision step walks a cell's pairs in windows of 64: cells of
one pair, of one window more or less, of whole and broken windows, and above the
shared-memory size, with few and many collections, against the oracle bit for
bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# pairs: 1, 3, 55, 66, 78 (around one window), 528, 2016 (a couple may straddle
# rows), ..., 32640 and 32896 (the largest in shared memory, the first beyond)
COUNTS = (2, 3, 11, 12, 13, 33, 64, 65, 129, 255, 256, 257)


def _state(rain):
    from conftest import with_rain
    from lacmopy_gb300 import synthetic
    n = sum(COUNTS)
    st = synthetic.make_icmw_state(Nx=4, Nz=3, no_spcm=(40, 60), seed=5, kernel_type="Hall_Bott",
                                   r_tot=12.5E-3, drizzle_fraction=0.2)
    assert st["xi"].size >= n
    for k in ("pos", "vel", "rel_pos", "cells"):
        st[k] = np.ascontiguousarray(st[k][:, :n])
    for k in ("m_w", "m_s", "xi", "T_p", "active_ids", "id_list", "mode"):
        st[k] = st[k][:n].copy()
    order = np.random.default_rng(3).permutation(n)
    cell = np.repeat(np.arange(len(COUNTS)), COUNTS)[order]
    st["cells"] = np.array([cell // 3, cell % 3], dtype=np.int64)
    return with_rain(st, rain) if rain else st


def _compare(ds, st, xi, mw, ms, nc):
    out = ds.snapshot()
    assert np.array_equal(out["no_cols"], nc)
    for k, v in (("xi", xi), ("m_w", mw), ("m_s", ms)):
        assert np.array_equal(out[k], v), k


@pytest.mark.parametrize("boost,rain", [(1.0, 0), (60.0, 0), (1.0, 2), (3000.0, 1)])
@pytest.mark.parametrize("draws", ["philox", "injected"])
def test_windows_match_oracle(oracle_cr, draws, boost, rain):
    from lacmopy_gb300 import DeviceState
    st = _state(rain)
    st["dt_col_over_dV"] = st["dt_col_over_dV"] * boost
    xi, mw, ms = st["xi"].copy(), st["m_w"].copy(), st["m_s"].copy()
    nc, cs = np.zeros(2, np.int64), np.zeros(1, np.int64)
    T, args = st["grid_scalar_fields"][0], (st["dt_col_over_dV"], st["E_col_grid"],
                                            st["no_kernel_bins"], st["R_kernel_low_log"],
                                            st["bin_factor_R_log"], nc, "AS")
    if draws == "philox":
        ds = DeviceState(st, draws="philox", seed=41)
        ds.collision_step()
        oracle_cr.collision_step_all_cells_philox(xi, mw, ms, st["vel"], T, st["cells"],
                                                  st["grid_no_cells"], *args, 41, cs)
    else:
        # some draws at and around zero, where the screens' lower bound ends
        rng = np.random.default_rng(9)
        u = rng.random(sum(c * (c - 1) // 2 for c in COUNTS))
        sel = rng.random(u.size) < 0.02
        u[sel] = rng.choice([0.0, 1e-300, 1e-12, 5e-8, 7e-8, 1.0 - 2.0 ** -53], sel.sum())
        ds = DeviceState(st, draws="philox")
        ds.collision_step(u)
        oracle_cr.collision_step_Ecol_grid_R_all_cells_2D_multicomp_np(
            xi, mw, ms, st["vel"], T, st["cells"], st["grid_no_cells"], *args, u)
    assert boost * (1 + rain) == 1.0 or nc.sum() > 0
    _compare(ds, st, xi, mw, ms, nc)


def test_efficiency_table_with_nan(oracle_cr):
    """A NaN in a row of the efficiency table hides the values before it from a
    maximum taken in column order; the first screen must not rely on that one."""
    from lacmopy_gb300 import DeviceState
    st = _state(2)
    E = st["E_col_grid"] = st["E_col_grid"].copy()
    E[:, -1] = np.nan
    E[::2, 3] = np.nan
    xi, mw, ms = st["xi"].copy(), st["m_w"].copy(), st["m_s"].copy()
    nc, cs = np.zeros(2, np.int64), np.zeros(1, np.int64)
    ds = DeviceState(st, draws="philox", seed=17)
    ds.collision_step()
    oracle_cr.collision_step_all_cells_philox(
        xi, mw, ms, st["vel"], st["grid_scalar_fields"][0], st["cells"], st["grid_no_cells"],
        st["dt_col_over_dV"], E, st["no_kernel_bins"], st["R_kernel_low_log"],
        st["bin_factor_R_log"], nc, "AS", 17, cs)
    assert nc.sum() > 0
    _compare(ds, st, xi, mw, ms, nc)
