"""The f64 translation products on the FP64 tensor path: runs of one table with fewer rows
than a fragment (16), more than a block's warps take at once, several vectors, and orders
whose slots end inside a group of eight or a K-step (p even), fill them (p = 3, 7, 11) or
split the table over two blocks (p = 12), against the oracle; the complex form against the
mixed evaluation, whose translations run on other kernels."""
import numpy as np
import pytest

import fmm_b200 as F

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))


# 1e-12: the f64 path's bound against the oracle on the same tree and order
@pytest.mark.parametrize("p,n,leaf,m", [(3, 400, 6, 1), (4, 400, 6, 5), (7, 9000, 16, 3), (8, 9000, 16, 1),
                                        (8, 700, 4, 17), (11, 2000, 12, 2), (12, 2000, 12, 3)])
def test_products_match_oracle(oracle, p, n, leaf, m):
    x, q = oracle.point_sets("sphere", n, 3 + p)
    qs = np.stack([q * (1.0 + 0.5 * v) + v * q[::-1] for v in range(m)], axis=1)
    fmm = F.FmmBuilder(p).vectors(m).max_points_per_leaf(leaf).build(x)
    out = fmm.evaluate(qs)
    for v in {0, m // 2, m - 1}:
        phi, _ = oracle.fmm(x, np.ascontiguousarray(qs[:, v]), x, p, leaf, threads=8)
        assert rel(out.potential[v], phi[0]) < 1e-12
    lv = fmm.evaluate_levels(qs)
    assert np.array_equal(lv.potential, out.potential)
    fmm.close()


# 5e-6: f32 expansions and pairs (the Helmholtz mixed form's bound)
@pytest.mark.parametrize("p,m", [(3, 1), (5, 2), (6, 1), (8, 2), (9, 1)])
def test_complex_products_match_mixed(oracle, p, m):
    x, _ = oracle.point_sets("sphere", 5000, 40 + p)
    rng = np.random.default_rng(p)
    q = rng.standard_normal((len(x), m)) + 1j * rng.standard_normal((len(x), m))
    out = []
    for precision in ("f64", "mixed"):
        fmm = F.FmmBuilder(p).gradients().vectors(m).max_points_per_leaf(16).precision(precision).build(x)
        out.append(fmm.helmholtz_evaluate(4.0, q))
        fmm.close()
    assert rel(out[1].potential, out[0].potential) < 5e-6
    assert rel(out[1].gradient, out[0].gradient) < 5e-6
