"""Levels run as one chain launch (few children x vectors) and as launches over the device give
the same floats: eight vectors move levels of a tree from one form to the other, at orders
whose tables fit the chain and not (f64 p = 12); the Helmholtz form; both against the level
calls, which run every level on its own."""
import numpy as np
import pytest

import fmm_b200 as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("p,n,leaf", [(3, 9000, 8), (6, 9000, 12), (8, 6000, 16), (12, 2500, 16)])
def test_chain_and_wide_levels_same_floats(oracle, precision, p, n, leaf):
    x, q = oracle.point_sets("sphere", n, p)
    b = F.FmmBuilder(p).max_points_per_leaf(leaf).precision(precision)
    one = b.vectors(1).build(x)
    want = one.evaluate(q)
    lv = one.evaluate_levels(q)
    assert np.array_equal(lv.potential, want.potential)
    one.close()
    many = b.vectors(8).build(x)
    got = many.evaluate(np.stack([q * (v + 1.0) for v in range(8)], axis=1))
    assert np.array_equal(got.potential[0], want.potential[0])
    assert np.array_equal(got.potential[3], 4.0 * want.potential[0])  # a power of two: exact
    many.close()


@pytest.mark.parametrize("precision,p", [("f64", 4), ("f64", 8), ("mixed", 4), ("mixed", 10), ("mixed", 12)])
def test_helmholtz_chain_and_wide_levels_same_floats(oracle, precision, p):
    x, q = oracle.point_sets("sphere", 5000, p)
    z = q + 1j * q[::-1]
    b = F.FmmBuilder(p).gradients().max_points_per_leaf(16).precision(precision)
    one = b.vectors(1).build(x)
    want = one.helmholtz_evaluate(5.0, z)
    one.close()
    two = b.vectors(5).build(x)
    got = two.helmholtz_evaluate(5.0, np.stack([z * (v + 1.0) for v in range(5)], axis=1))
    scale = np.linalg.norm(want.potential)
    # the near field and the tensor-core M2L of several vectors run on other kernels in the
    # mixed form: 5e-6 there (f32 pairs), the same floats in f64
    tol = 0.0 if precision == "f64" else 5e-6
    assert np.linalg.norm(got.potential[0] - want.potential[0]) <= tol * scale
    two.close()
