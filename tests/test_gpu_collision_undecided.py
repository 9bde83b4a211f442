"""Per-pair collision steps with many pairs that the FP32 bounds cannot decide and
that change nothing (multiplicities below zero, as multiple collections can leave
them, or NaN velocities): a cell gives up its event chain for the anti-diagonals
after enough of them.  Few and many in a cell, with and without collections among
them, in shared memory and above it, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boost", [1.0, 300.0])
@pytest.mark.parametrize("share", [0.01, 0.05, 0.4, 1.0])
@pytest.mark.parametrize("kind", ["negative", "nan"])
@pytest.mark.parametrize("draws", ["philox", "thinned"])
def test_undecided_pairs(oracle_cr, draws, kind, share, boost):
    from lacmopy_gb300 import DeviceState
    from test_gpu_collision_windows import _compare, _state
    st = _state(1)
    st["dt_col_over_dV"] = st["dt_col_over_dV"] * boost
    rng = np.random.default_rng(8)
    sel = rng.random(st["xi"].size) < share
    if kind == "negative":
        st["xi"][sel] = -rng.random(sel.sum())
    else:
        st["vel"][0, sel] = np.nan
    xi, mw, ms = st["xi"].copy(), st["m_w"].copy(), st["m_s"].copy()
    nc, cs = np.zeros(2, np.int64), np.zeros(1, np.int64)
    ds = DeviceState(st, draws=draws, seed=41)
    ds.collision_step()
    oracle_cr.collision_step_all_cells_philox(
        xi, mw, ms, st["vel"], st["grid_scalar_fields"][0], st["cells"], st["grid_no_cells"],
        st["dt_col_over_dV"], st["E_col_grid"], st["no_kernel_bins"], st["R_kernel_low_log"],
        st["bin_factor_R_log"], nc, "AS", 41, cs, thin=draws == "thinned")
    assert share == 1.0 or nc.sum() > 0
    _compare(ds, st, xi, mw, ms, nc)
