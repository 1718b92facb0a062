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


# P2L rows of about 17,000 sources of one sign, far field alone, in f32 against f64 at the same order:
# f32's roundings are 1.7e-7 (p = 6, 2 vectors) to 2.8e-7 (p = 11) when a row's sum adds next to nothing
# to them, 5.5e-7 to 6.5e-7 when it runs over the sources one after another
@pytest.mark.parametrize("p,m,tol", [(6, 2, 3e-7), (6, 16, 3e-7), (11, 1, 4e-7)])
def test_long_rows_keep_their_precision(p, m, tol):
    rng = np.random.default_rng(1)
    x, t = rng.random((57000, 3)), rng.random((230000, 3))
    x[:, 0] *= 0.5  # coarse leaves of about 1,800 sources beside finer ones of targets
    t[:, 0] = 0.5 + 0.5 * t[:, 0]
    q = rng.random((len(x), m))
    out = []
    for precision in ("f64", "mixed"):
        fmm = F.FmmBuilder(p).vectors(m).max_points_per_leaf(2100).precision(precision).build(x, t)
        assert fmm.info()["x_pairs"] > 500
        fmm.set_kinds(2)
        out.append(fmm.evaluate(q).potential[:, (t[:, 0] > 0.625) & (t[:, 0] < 0.75)])
        fmm.close()
    err = (out[1] - out[0]) / out[0]
    assert np.sqrt((err * err).mean(axis=1)).max() < tol
