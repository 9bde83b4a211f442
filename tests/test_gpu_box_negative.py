"""Box-model steps of SIPs with multiplicities of zero and below, as multiple
collections can leave them: the partner of such a SIP gains multiplicity in a
collection.  Against the oracle bit for bit, below and above the pair count that
one CTA screens itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["golovin", "kgrid", "ecol"])
@pytest.mark.parametrize("n", [3, 40, 128, 129, 600])
@pytest.mark.parametrize("share,value", [(0.02, -1.0), (0.3, -1.0), (0.3, 0.0), (0.1, -1e6)])
def test_negative_multiplicities(oracle_cr, kind, n, share, value):
    from lacmopy_gb300 import collision as C
    from test_gpu_box import _case, _draws, _run
    seen = 0
    for dtdv in (3.0, 60.0, 1000.0):
        a, tab = _case(kind, n, 3, False)
        rng = np.random.default_rng(n)
        sel = rng.random(n) < share
        sel[rng.integers(n)] = True
        a[0][sel] = value if value == -1e6 else value * a[0][sel]
        b = [v.copy() for v in a]
        na, nb = np.zeros(2, np.int64), np.zeros(2, np.int64)
        for q in range(3):
            u = _draws(n, 10 * n + q)
            _run(C, kind, a, dtdv, na, tab, draws=u)
            _run(oracle_cr, kind, b, dtdv, nb, tab, draws=u)
        assert np.array_equal(na, nb), (dtdv, na, nb)
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True), dtdv
        seen += int(na.sum())
    assert n == 3 or seen > 0
