"""An FMM on a plan given from outside (fmmgpu_upload_plan, the reference's
DeviceOperator::new on its own plan), needs a B200: -m gpu.  The library's plan exported
and uploaded again gives the library's bits (fused evaluation and level calls); the
oracle's plan (its tree and brute-force lists, boxes without sources kept in the rows)
gives the oracle FMM's result within 1e-12."""
import ctypes as C

import numpy as np
import pytest

import fmm_b200 as F
from tests.plan_arrays import oracle_plan

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_uploaded_library_plan_gives_the_same_bits(precision):
    rng = np.random.default_rng(8)
    x = rng.uniform(size=(20000, 3))
    q = rng.standard_normal(20000)
    own = F.FmmBuilder(6).gradients().max_points_per_leaf(32).precision(precision).build(x)
    arrays = own.plan_arrays()
    up = F.FmmBuilder(6).gradients().precision(precision).upload(arrays, x)
    a, b = own.evaluate(q), up.evaluate(q)
    assert np.array_equal(a.potential, b.potential) and np.array_equal(a.gradient, b.gradient)
    c = up.evaluate_levels(q)
    assert np.array_equal(c.potential, a.potential) and np.array_equal(c.gradient, a.gradient)


def test_uploaded_oracle_plan_matches_the_oracle_fmm(oracle):
    x, q = oracle.point_sets("sphere", 12000, 9)
    arrays = oracle_plan(oracle, x, x, 24)
    up = F.FmmBuilder(6).gradients().precision("f64").upload(arrays, x)
    out = up.evaluate(q)
    phi, g = oracle.fmm(x, q, x, 6, 24, gradients=True, threads=8)
    assert rel(out.potential, phi) < 1e-12 and rel(out.gradient, g) < 1e-12


def nan_holes(cuda, sizes):
    """Device buffers of these sizes filled with NaN, every other one freed again, so that the
    next allocations of such a size take memory that holds NaN; the ones kept."""
    held = []
    for size in sizes:
        ptrs = []
        for _ in range(200):
            ptr = C.c_uint64()
            assert cuda.cuMemAlloc_v2(C.byref(ptr), C.c_size_t(size)) == 0
            assert cuda.cuMemsetD8_v2(ptr, C.c_ubyte(255), C.c_size_t(size)) == 0
            ptrs.append(ptr)
        assert cuda.cuCtxSynchronize() == 0
        for ptr in ptrs[1::2]:
            assert cuda.cuMemFree_v2(ptr) == 0
        held += ptrs[::2]
    return held


@pytest.mark.parametrize("precision,p,m", [("f64", 4, 1), ("f64", 9, 2), ("mixed", 4, 1), ("mixed", 10, 3)])
def test_x_rows_of_leaves_without_sources_add_nothing(precision, p, m):
    """X rows that name only leaves without a source (an uploaded plan may) change no bit of the
    Laplace or the Helmholtz evaluation, whatever the device memory held before."""
    cuda = C.CDLL("libcuda.so.1")
    rng = np.random.default_rng(21)
    x = 0.45 * rng.random((3000, 3))  # sources in one corner, targets everywhere
    t = np.concatenate([rng.random((4000, 3)), 0.2 + 0.02 * rng.random((2000, 3))])
    b = F.FmmBuilder(p).gradients().vectors(m).precision(precision).max_points_per_leaf(24)
    plan = b.plan(x, t).plan_arrays()
    level = (plan["keys"] & np.uint64(0x7FFF)).astype(int)
    leaf_level = level[np.flatnonzero(plan["is_leaf"])]
    empty = np.diff(plan["source_offsets"].astype(np.int64)) == 0
    rows = [list(plan["x"][plan["x_rows"][i]:plan["x_rows"][i + 1]]) for i in range(len(level))]
    added = 0
    for i, row in enumerate(rows):
        pick = np.flatnonzero(empty & (leaf_level == level[i] - 1))
        if level[i] >= 2 and not row and len(pick):
            row.append(int(pick[i % len(pick)]))
            added += 1
    assert added > 100
    more = dict(plan)
    more["x_rows"] = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(plan["x_rows"].dtype)
    more["x"] = np.array([v for r in rows for v in r], dtype=plan["x"].dtype)
    q = rng.standard_normal((len(x), m))
    z = q + 1j * rng.standard_normal((len(x), m))
    b.upload(plan, x, t).close()  # (the device's context is current from here on)
    row_bytes = m * ((p + 1) ** 2 + 3) // 4 * 4 * (8 if precision == "f64" else 4)
    out = []
    for arrays in (plan, more):
        held = nan_holes(cuda, [row_bytes * len(level), 2 * row_bytes * len(level)])
        fmm = b.upload(arrays, x, t)
        a, h = fmm.evaluate(q), fmm.helmholtz_evaluate(5.0, z)
        out.append((a.potential, a.gradient, h.potential, h.gradient))
        fmm.close()
        for ptr in held:
            assert cuda.cuMemFree_v2(ptr) == 0
    for want, got in zip(*out):
        assert np.isfinite(want).all() and np.array_equal(got, want)
