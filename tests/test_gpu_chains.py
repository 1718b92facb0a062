"""Levels run as one chain launch (few children x vectors) and as launches over the device give
the same floats: eight vectors a pass move levels of a tree from one form to the other, at orders
whose tables fit the chain and not (f64 p = 12); the Helmholtz form; both against the level
calls, which run every level on its own."""
import numpy as np
import pytest

import fmm_b200 as F

pytestmark = pytest.mark.gpu


CHAIN_ROWS = 1024  # children x vectors of a level up to which it stays in a chain


def both_forms(fmm, few, many):
    """Whether some level of the tree (boxes over a source, below the root) stays in a chain with
    `few` vectors a pass and runs wide with `many`."""
    plan = fmm.plan_arrays()
    keys = plan["keys"].astype(np.uint64)
    level = (keys & np.uint64(0x7FFF)).astype(int)
    leaves = np.flatnonzero(plan["is_leaf"])
    used = keys[leaves[np.diff(plan["source_offsets"].astype(np.int64)) > 0]]
    count = np.zeros(level.max() + 1, dtype=int)
    for l in range(level.max(), 0, -1):  # the used boxes of level l, then their parents
        at = (used & np.uint64(0x7FFF)) == l
        here = np.unique(used[at])
        count[l] = len(here)
        shift = np.uint64(15 + 3 * (16 - (l - 1)))
        used = np.concatenate([used[~at], ((here >> shift) << shift) | np.uint64(l - 1)])
    return any(c * few <= CHAIN_ROWS < c * many for c in count[3:])


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("p,n,leaf", [(3, 9000, 8), (6, 9000, 12), (8, 6000, 16), (12, 2500, 16)])
def test_chain_and_wide_levels_same_floats(oracle, precision, p, n, leaf):
    x, q = oracle.point_sets("sphere", n, p)
    qs = np.stack([q * (v + 1.0) for v in range(8)], axis=1)
    b = F.FmmBuilder(p).vectors(8).max_points_per_leaf(leaf).precision(precision)
    one = b.vectors_per_pass(1).build(x)  # a vector a pass: small levels in chains
    want = one.evaluate(qs)
    one.close()
    many = b.vectors_per_pass(8).build(x)  # eight rows a child: the same levels wide
    got = many.evaluate(qs)
    assert np.array_equal(got.potential, want.potential)
    lv = many.evaluate_levels(qs)
    assert np.array_equal(lv.potential, want.potential)
    assert both_forms(many, 1, 8)
    many.close()


@pytest.mark.parametrize("precision,p", [("f64", 4), ("f64", 8), ("mixed", 4), ("mixed", 10), ("mixed", 12)])
def test_helmholtz_chain_and_wide_levels_same_floats(oracle, precision, p):
    x, q = oracle.point_sets("sphere", 5000, p)
    z = q + 1j * q[::-1]
    b = F.FmmBuilder(p).gradients().max_points_per_leaf(16).precision(precision)
    zs = np.stack([z * (v + 1.0) for v in range(5)], axis=1)
    b = b.vectors(5)
    one = b.vectors_per_pass(1).build(x)
    want = one.helmholtz_evaluate(5.0, zs)
    one.close()
    two = b.vectors_per_pass(5).build(x)
    got = two.helmholtz_evaluate(5.0, zs)
    # the near field of one vector runs on another kernel in the mixed form: 5e-6 there (f32
    # pairs; the levels' floats are compared below), the same floats in f64
    tol = 0.0 if precision == "f64" else 5e-6
    assert np.linalg.norm(got.potential - want.potential) <= tol * np.linalg.norm(want.potential)
    two.close()


@pytest.mark.parametrize("precision,p", [("f64", 4), ("f64", 8), ("mixed", 4), ("mixed", 10), ("mixed", 12)])
def test_helmholtz_levels_same_floats_whatever_the_pass(oracle, precision, p):
    x, q = oracle.point_sets("sphere", 5000, p)
    z = q + 1j * q[::-1]
    b = F.FmmBuilder(p).gradients().max_points_per_leaf(16).precision(precision).vectors(8)
    zs = np.stack([z * (v + 1.0) for v in range(8)], axis=1)
    few = b.vectors_per_pass(2).build(x)  # two, not one: the near field's kernel is then the same
    assert both_forms(few, 2, 8)
    want = few.helmholtz_evaluate(5.0, zs)
    few.close()
    many = b.vectors_per_pass(8).build(x)
    got = many.helmholtz_evaluate(5.0, zs)
    assert np.array_equal(got.potential, want.potential) and np.array_equal(got.gradient, want.gradient)
    many.close()


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_helmholtz_leaf_sums_of_many_vectors(oracle, precision):
    """P2M and P2L stage 64 vectors' charges at a time, and a tile of the mixed M2L holds 128 columns, two
    a vector: 65 to 130 vectors a pass give the floats of 10 a pass."""
    x, q = oracle.point_sets("sphere", 2500, 3)
    m = 130
    z = np.stack([(q + 1j * q[::-1]) * (v + 1.0) * (-1) ** v for v in range(m)], axis=1)
    b = F.FmmBuilder(3).gradients().max_points_per_leaf(12).precision(precision).vectors(m)
    out = []
    for passes in (10, 65, 130):
        fmm = b.vectors_per_pass(passes).build(x)
        assert fmm.info()["x_pairs"] > 0
        if precision == "f64":
            assert fmm.info()["vectors_per_pass"] == passes
        o = fmm.helmholtz_evaluate(3.0, z)
        out.append((o.potential, o.gradient))
        fmm.close()
    for potential, gradient in out[1:]:
        assert np.array_equal(potential, out[0][0]) and np.array_equal(gradient, out[0][1])


@pytest.mark.parametrize("p,m,few", [(8, 49, 7), (8, 67, 1), (10, 33, 3)])
def test_helmholtz_vectors_beyond_one_tile(oracle, p, m, few):
    """Twice the vectors are more than a tile's columns (96 at p = 8, 64 at p = 10)."""
    x, q = oracle.point_sets("sphere", 2500, 4)
    z = np.stack([(q + 1j * q[::-1]) * (v + 1.0) for v in range(m)], axis=1)
    b = F.FmmBuilder(p).max_points_per_leaf(40).precision("mixed").vectors(m)
    one, many = b.vectors_per_pass(few).build(x), b.vectors_per_pass(m).build(x)
    assert many.info()["vectors_per_pass"] == m
    want, got = one.helmholtz_evaluate(3.0, z).potential, many.helmholtz_evaluate(3.0, z).potential
    # a vector a pass has another near-field kernel in the mixed form
    tol = 5e-6 if few == 1 else 0.0
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
    one.close()
    many.close()
