"""Box-model collision steps against the oracle bit for bit, at the sizes where
the step changes its course: pairs screened by one CTA or by the whole GPU
(8128 pairs of 128 SIPs, 8256 of 129), the largest SIP counts, and from no
collection to so many that the anti-diagonal schedule takes the step at its start
or in the middle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sips(n, seed, equal=False):
    rng = np.random.default_rng(seed)
    m_mean = 4.18879e3 * 9.3 ** 3
    edges = np.exp(np.linspace(np.log(1e-3 * m_mean), np.log(30.0 * m_mean), n + 1))
    m = edges[:-1] + rng.random(n) * np.diff(edges)
    xi = 1e15 / m_mean * np.exp(-m / m_mean) / m_mean * np.diff(edges) + 1.0
    if equal:   # pairs of equal multiplicity split
        xi[::2] = xi[0]
    perm = rng.permutation(n)
    return xi[perm], m[perm]


def _draws(n, seed, edges=True):
    rng = np.random.default_rng(seed)
    u = rng.random(n * (n - 1) // 2)
    if edges:
        k = min(u.size, 40)
        sel = rng.choice(u.size, size=k, replace=False)
        u[sel] = rng.choice([0.0, 1e-300, 5e-8, 7e-8, 1.0 - 2.0 ** -53], k)
    return u


def _tables():
    from lacmopy_gb300.tables import load_kernel_data_Ecol
    E, _, _, _, lo, bl, nb = load_kernel_data_Ecol("Hall_Bott")
    return E, nb, lo, bl


def _run(mod, kind, sips, dtdv, nc, tab, **kw):
    draws = kw.pop("draws")
    if kind == "golovin":
        mod.collision_step_Golovin_np(sips[0], sips[1], dtdv, nc, draws=draws, **kw)
    elif kind == "kgrid":
        K, nb, lo, bl = tab
        mod.collision_step_kernel_grid_m_np(sips[0], sips[1], dtdv, K, nb, lo, bl, nc, draws=draws,
                                            **kw)
    else:
        E, nb, lo, bl = tab
        mod.collision_step_Ecol_grid_R_np(*sips, dtdv, E, nb, lo, bl, nc, draws=draws, **kw)


def _case(kind, n, seed, equal):
    xi, m = _sips(n, seed, equal)
    if kind == "golovin":
        return [xi, m], None
    if kind == "kgrid":   # a sum kernel on a coarse mass grid, with zeros
        nb, lo, bl = 40, np.log(m.min()) - 0.1, (np.log(m.max()) - np.log(m.min())) / 38
        g = np.exp(lo + bl * np.arange(nb))
        K = 1.5e-18 * (g[:, None] + g[None, :])
        K[5] = 0.0
        return [xi, m], (K, nb, lo, bl)
    R = (m / 4.18879e3) ** (1.0 / 3.0)
    vel = 1.2e-4 * R * R
    return [xi, m, R, vel, np.full(n, 1000.0)], _tables()


def _check(orc, kind, n, dtdv, draws, equal=False):
    from lacmopy_gb300 import collision as C
    a, tab = _case(kind, n, 3, equal)
    b = [v.copy() for v in a]
    na, nb_ = np.zeros(2, np.int64), np.zeros(2, np.int64)
    for _ in range(2):
        _run(C, kind, a, dtdv, na, tab, draws=draws)
        _run(orc, kind, b, dtdv, nb_, tab, draws=draws)
    assert np.array_equal(na, nb_), (na, nb_)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    return int(na.sum())


@pytest.mark.parametrize("kind", ["golovin", "kgrid", "ecol"])
@pytest.mark.parametrize("n", [2, 3, 64, 128, 129, 1000])
def test_box_sizes(oracle_cr, kind, n):
    # from a few collections a step to more than one per SIP
    for dtdv in (1.0, 30.0, 1000.0):
        _check(oracle_cr, kind, n, dtdv, _draws(n, n))
    _check(oracle_cr, kind, n, 30.0, _draws(n, n + 1, edges=False), equal=True)


@pytest.mark.parametrize("kind,n", [("golovin", 8192), ("kgrid", 8192), ("ecol", 4096)])
def test_box_largest(oracle_cr, kind, n):
    assert _check(oracle_cr, kind, n, 3.0, _draws(n, 1)) > 0


@pytest.mark.parametrize("kind,n", [("golovin", 65), ("golovin", 1001), ("ecol", 129)])
def test_box_philox(oracle_cr, kind, n):
    u = oracle_cr.philox_uniform(17, np.arange(n * (n - 1) // 2),
                                 np.full(n * (n - 1) // 2, (5 << 32) | 2))
    from lacmopy_gb300 import collision as C
    a, tab = _case(kind, n, 8, False)
    b = [v.copy() for v in a]
    na, nb_ = np.zeros(2, np.int64), np.zeros(2, np.int64)
    _run(C, kind, a, 40.0, na, tab, draws="philox", seed=17, step=(5 << 32) | 2)
    _run(oracle_cr, kind, b, 40.0, nb_, tab, draws=u)
    assert na.sum() > 0 and np.array_equal(na, nb_)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
