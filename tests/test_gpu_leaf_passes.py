"""P2M, P2L, L2P and M2P against the oracle where their lanes are not full: leaves of more and
of fewer sources than a warp's 32, X lists of several leaves, one to seventeen vectors (passes
of 1, 4 and 16 vectors and their remainders), targets times vectors above a warp's lanes."""
import numpy as np
import pytest

import fmm_b200 as F

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))


# 1e-12 and 2e-6: the f64 path's and the mixed form's bounds against the oracle
@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("mixed", 2e-6)])
@pytest.mark.parametrize("p,leaf,m", [(3, 6, 1), (4, 48, 2), (6, 12, 5), (8, 40, 17), (11, 24, 3), (12, 80, 4)])
def test_leaf_passes_match_oracle(oracle, precision, tol, p, leaf, m):
    rng = np.random.default_rng(p)
    x = np.concatenate([oracle.point_sets("sphere", 2500, p)[0], 0.9 + 0.02 * rng.random((700, 3))])
    t = np.concatenate([x[::3] + 1e-3, rng.random((500, 3))])
    q = rng.standard_normal((len(x), m))
    fmm = F.FmmBuilder(p).gradients().vectors(m).max_points_per_leaf(leaf).precision(precision).build(x, t)
    info = fmm.info()
    assert info["x_pairs"] > 0 and info["w_pairs"] > 0
    out = fmm.evaluate(q)
    for v in {0, m - 1}:
        phi, g = oracle.fmm(x, np.ascontiguousarray(q[:, v]), t, p, leaf, gradients=True, threads=8)
        assert rel(out.potential[v], phi[0]) < tol and rel(out.gradient[v], g[0]) < tol
    lv = fmm.evaluate_levels(q)
    assert np.array_equal(lv.potential, out.potential) and np.array_equal(lv.gradient, out.gradient)
    fmm.close()
