"""FP64 sub-steps of SIPs without solute (m_s = 0), whose masses lie outside the
two-float range: whole warps of them, a few among others, and more of them in a
block than its queue holds.

Tolerances: 1e-10 is the product's stated agreement; velocities are one rounding
of a sum of terms no larger than 20 m/s, 1e-12 m/s absolute.  Two runs give the
same bits: which SIPs find room in the queue must not show."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, share, sol, seed=3):
    from lacmopy_gb300 import synthetic
    rng = np.random.default_rng(seed)
    st = synthetic.make_icmw_state(Nx=7, Nz=5, no_spcm=(1, 1), seed=4, r_tot=12.5E-3)
    dx, dz = st["grid_steps"]
    i, j = rng.integers(0, 7, n), rng.integers(1, 5, n)
    rel = rng.uniform(0.1, 0.9, (2, n))
    R = np.exp(rng.uniform(np.log(5.0), np.log(60.0), n))
    m_s = 4.18879 * 1774.0 * np.exp(rng.uniform(np.log(2e-2), np.log(2e-1), n)) ** 3
    m_s[rng.random(n) < share] = 0.0
    st.update(pos=np.array([(i + rel[0]) * dx, (j + rel[1]) * dz]),
              vel=rng.normal(0.0, 0.3, (2, n)), cells=np.array([i, j], dtype=np.int64),
              rel_pos=rel, m_w=4.18879e3 * R ** 3, m_s=m_s, xi=rng.uniform(1e3, 1e6, n),
              T_p=np.ones(n), active_ids=np.full(n, True), id_list=np.arange(n), solute_type=sol)
    st["grid_scalar_fields"][6] = 1.002
    return st


def _copy(st):
    return {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in st.items()}


def _sub_step(mod, st):
    mod.propagate_particles_subloop_step_np(
        st["grid_scalar_fields"], st["grid_mat_prop"], st["grid_velocity"], st["grid_no_cells"],
        st["grid_ranges"], st["grid_steps"], st["pos"], st["vel"], st["cells"], st["rel_pos"],
        st["m_w"], st["m_s"], st["xi"], st["water_removed"], None, st["active_ids"], st["T_p"],
        st["solute_type"], st["delta_m_l"], 0.1, 0.1, 3, 9.80665)


# 1.5 million SIPs: some 2500 to a block where four blocks an SM are resident, half
# or all of them without solute, against a queue of 1024
@pytest.mark.parametrize("n,share", [(33, 1.0), (3000, 1.0), (3000, 0.1), (100000, 0.5),
                                     (1500000, 0.5), (1500000, 0.97)])
@pytest.mark.parametrize("sol", ["AS", "NaCl"])
def test_sub_step_without_solute(oracle_nb, n, share, sol):
    from lacmopy_gb300 import integration as I
    a = _state(n, share, sol)
    again, ref = _copy(a), _copy(a)
    _sub_step(I, a)
    _sub_step(I, again)
    _sub_step(oracle_nb, ref)
    for k in ("m_w", "vel", "pos", "delta_m_l"):
        assert np.array_equal(a[k], again[k]), k
    assert np.array_equal(a["cells"], ref["cells"])
    np.testing.assert_allclose(a["m_w"], ref["m_w"], rtol=1e-10)
    np.testing.assert_allclose(a["vel"], ref["vel"], rtol=1e-10, atol=1e-12)
    np.testing.assert_allclose(a["delta_m_l"], ref["delta_m_l"], rtol=1e-10)
