"""The integer sums of the FP64 sub-step (condensed mass per cell, water removed at
the ground): many kilograms in a sub-step, products far below one fg, and both
together, for states whose words hold 42 bits (up to 2^20 SIPs) and fewer.

Tolerances: with the masses the sub-step wrote, dm xi is the product the kernel
formed (steps below an eighth of the mass store m_w + dm itself), so the reference
is the exactly rounded sum of the same products (math.fsum).  The kernel's sum is
within 0.8 of a last place, its factor 1e-18 rounds once more and so does the
reference's: 2 last places, 4.5e-16; products below 2^-12 fg add 2^-65 fg each.
Against the oracle: 1e-10, the product's stated agreement; removed water is a sum
of positive terms, 1e-12."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, cell=(2, 3), R=(10.0, 40.0), seed=3):
    """n cloud drops (radii R, um) in one cell of a 7 x 5 grid, falling slowly."""
    from lacmopy_gb300 import synthetic
    rng = np.random.default_rng(seed)
    st = synthetic.make_icmw_state(Nx=7, Nz=5, no_spcm=(1, 1), seed=4, r_tot=12.5E-3)
    dx, dz = st["grid_steps"]
    i, j = np.full(n, cell[0]), np.full(n, cell[1])
    pos = np.array([(i + rng.uniform(0.2, 0.8, n)) * dx, (j + rng.uniform(0.2, 0.8, n)) * dz])
    m_s = 4.18879 * 1774.0 * np.exp(rng.uniform(np.log(2e-2), np.log(2e-1), n)) ** 3
    m_w = 4.18879e3 * np.exp(rng.uniform(np.log(R[0]), np.log(R[1]), n)) ** 3
    st.update(pos=pos, vel=np.zeros((2, n)), cells=np.array([i, j], dtype=np.int64),
              rel_pos=np.array([pos[0] / dx - i, pos[1] / dz - j]), m_w=m_w, m_s=m_s,
              xi=np.ones(n), T_p=np.ones(n), active_ids=np.full(n, True), id_list=np.arange(n),
              solute_type="AS")
    st["grid_scalar_fields"][6][cell] = 1.01   # supersaturated: every drop grows
    return st


def _copy(st):
    return {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in st.items()}


def _sub_step(mod, st, dt=0.1):
    mod.propagate_particles_subloop_step_np(
        st["grid_scalar_fields"], st["grid_mat_prop"], st["grid_velocity"], st["grid_no_cells"],
        st["grid_ranges"], st["grid_steps"], st["pos"], st["vel"], st["cells"], st["rel_pos"],
        st["m_w"], st["m_s"], st["xi"], st["water_removed"], None, st["active_ids"], st["T_p"],
        st["solute_type"], st["delta_m_l"], dt, dt, 3, 9.80665)


def _growth(st):
    """dm of every SIP in the sub-step (it does not depend on xi)."""
    from lacmopy_gb300 import integration as I
    a = _copy(st)
    _sub_step(I, a)
    dm = a["m_w"] - st["m_w"]
    assert (np.abs(dm) < 0.125 * st["m_w"]).all() and (dm != 0).all()
    return dm


@pytest.mark.parametrize("n,kg", [(64, 0.6), (40, 1.0), (130, 0.01), ((1 << 20) + 77, 0.9)])
def test_many_kilograms_condensed_in_a_cell(oracle_nb, n, kg):
    from lacmopy_gb300 import integration as I
    a = _state(n)
    dm = _growth(a)
    a["xi"] = kg * 1e18 / np.abs(dm)
    b = _copy(a)
    _sub_step(I, a)
    want = math.fsum(dm * a["xi"]) * 1e-18
    assert want > 0.8 * n * kg
    got = a["delta_m_l"][2, 3]
    assert abs(got - want) <= 4.5e-16 * want
    assert np.count_nonzero(a["delta_m_l"]) == 1
    if n < 1000:
        _sub_step(oracle_nb, b)
        np.testing.assert_allclose(a["delta_m_l"], b["delta_m_l"], rtol=1e-10, atol=0)


@pytest.mark.parametrize("n,kg", [(100, 1.0), (33, 1.1), ((1 << 20) + 5, 0.3)])
def test_many_kilograms_removed_at_the_ground(oracle_nb, n, kg):
    from lacmopy_gb300 import integration as I
    a = _state(n, cell=(4, 0))
    a["vel"][1] = -300.0
    a["pos"][1] = 1e-3 * a["grid_steps"][1]
    a["rel_pos"][1] = 1e-3
    a["xi"] = kg * 1e18 / a["m_w"]
    a["water_removed"][0] = 2.0
    b = _copy(a)
    _sub_step(I, a)
    assert not a["active_ids"].any()
    want = math.fsum(a["m_w"] * a["xi"])
    assert want > 0.9e18 * n * kg
    assert abs(a["water_removed"][0] - want) <= 4.5e-16 * want
    if n < 1000:
        _sub_step(oracle_nb, b)
        np.testing.assert_allclose(a["water_removed"], b["water_removed"], rtol=1e-12)


@pytest.mark.parametrize("n", [3, 500, (1 << 20) + 1])
@pytest.mark.parametrize("lo,hi", [(-9, -2), (-30, -20), (-20, 30), (25, 60), (58, 62)])
def test_products_of_any_size(n, lo, hi):
    """Products dm xi spread over 2^lo to 2^hi fg, a third of them negative."""
    from lacmopy_gb300 import integration as I
    a = _state(n, seed=n % 97)
    dm = _growth(a)
    rng = np.random.default_rng(5)
    a["xi"] = 2.0 ** rng.uniform(lo, hi, n) / np.abs(dm) * rng.choice([1.0, 1.0, -1.0], n)
    _sub_step(I, a)
    p = dm * a["xi"]
    want = math.fsum(p) * 1e-18
    small = np.count_nonzero(np.abs(p) < 2.0 ** -12) * 2.0 ** -65 * 1e-18
    assert abs(a["delta_m_l"][2, 3] - want) <= 4.5e-16 * abs(want) + small
