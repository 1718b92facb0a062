"""The Helmholtz FMM on the device (real k), against the oracle's Helmholtz FMM on the
same tree and lists and against the f64 direct sum (itself pinned to FMM3D's values in
test_gpu_helmholtz / test_helmholtz_oracle).  Needs a B200: -m gpu.

The oracle translates each pair by projection in absolute units while the device applies
per-level tables built by projection in box units (the same quadrature rule, another
evaluation order), so the f64 FMMs agree to rounding (within 1e-12 relative), not bit for
bit; the mixed form (f32 expansions and translations, complex64 near field) stays within
1e-5 of the f64 FMM."""
import numpy as np
import pytest

import fmm_b200 as F

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))


@pytest.fixture(scope="module")
def cloud():
    """1,000 points of a clipped Gaussian cluster: an adaptive tree of five levels (M2L on
    three, L2L on two, W and X lists) that the oracle's Python-level FMM runs in seconds."""
    rng = np.random.default_rng(31)
    x = np.clip(rng.normal(0.5, 0.12, (1000, 3)), 0.0, 1.0)
    q = rng.standard_normal(1000) + 1j * rng.standard_normal(1000)
    return x, q


def test_f64_matches_the_oracle_fmm(oracle, cloud):
    x, q = cloud
    k, p = 5.0, 6
    fmm = F.FmmBuilder(p).gradients().max_points_per_leaf(24).precision("f64").build(x)
    info = fmm.info()
    assert info["nlevels"] == 5 and info["w_pairs"] > 0 and info["x_pairs"] > 0
    out = fmm.helmholtz_evaluate(k, q)
    ophi, og = oracle.helmholtz_fmm(x, q, x, k, p, 24)
    ophi, og = ophi / (4 * np.pi), og / (4 * np.pi)
    ep, eg = rel(out.potential[0], ophi), rel(out.gradient[0], og)
    print(f"p={p}: f64 vs oracle FMM phi {ep:.2e} grad {eg:.2e}")
    assert ep < 1e-12 and eg < 1e-12  # measured 1.6e-15 and 1.3e-14
    fmm.close()


@pytest.mark.parametrize("p,tol", [(6, 2e-4), (10, 1e-5)])
def test_against_the_direct_sum(cloud, p, tol):
    x, q = cloud
    k = 5.0
    dphi, dg = F.helmholtz_direct_sum(k, x, q, x)
    for precision in ("f64", "mixed"):
        fmm = F.FmmBuilder(p).gradients().max_points_per_leaf(24).precision(precision).build(x)
        out = fmm.helmholtz_evaluate(k, q)
        ep, eg = rel(out.potential[0], dphi), rel(out.gradient[0], dg)
        print(f"p={p} {precision}: vs direct phi {ep:.2e} grad {eg:.2e}")
        assert ep < tol and eg < 10 * tol
        fmm.close()


def test_mixed_close_to_f64_and_repeatable():
    rng = np.random.default_rng(5)
    x = rng.uniform(0.0, 1.0, (20000, 3))
    q = rng.standard_normal((20000, 2)) + 1j * rng.standard_normal((20000, 2))
    k = 20.0
    outs = {}
    for precision in ("f64", "mixed"):
        fmm = F.FmmBuilder(8).gradients().vectors(2).max_points_per_leaf(48).precision(precision).build(x)
        a = fmm.helmholtz_evaluate(k, q)
        b = fmm.helmholtz_evaluate(k, q)  # tables kept for the same k: the same bits
        assert np.array_equal(a.potential, b.potential) and np.array_equal(a.gradient, b.gradient)
        outs[precision] = a
        fmm.close()
    ep = rel(outs["mixed"].potential, outs["f64"].potential)
    eg = rel(outs["mixed"].gradient, outs["f64"].gradient)
    print(f"mixed vs f64: phi {ep:.2e} grad {eg:.2e}")
    assert ep < 1e-5 and eg < 1e-5
    pick = np.arange(0, 20000, 97)
    dphi, _ = F.helmholtz_direct_sum(k, x, q[:, 1], x[pick], gradients=False)
    assert rel(outs["f64"].potential[1][pick], dphi) < 5e-4  # p = 8 at k = 20: measured 1.7e-4


def test_complex_wavenumber_is_refused(cloud):
    x, q = cloud
    fmm = F.FmmBuilder(6).max_points_per_leaf(32).build(x)
    with pytest.raises(F.FmmError) as e:
        fmm.helmholtz_evaluate(5.0 + 0.5j, q)
    assert e.value.status == 2
    fmm.close()


@pytest.mark.parametrize("precision", ["mixed", "f64"])
def test_complex64_call_is_the_complex128_call_rounded(cloud, precision):
    """fmmgpu_helmholtz_evaluate_f32: complex64 charges in, every complex64 output the
    complex128 call's result on the widened charges, rounded (real and imaginary parts)."""
    x, q = cloud
    q64 = q.astype(np.complex64)
    fmm = F.FmmBuilder(6).gradients().max_points_per_leaf(24).precision(precision).build(x)
    want = fmm.helmholtz_evaluate(5.0, q64.astype(np.complex128))
    got = fmm.helmholtz_evaluate(5.0, q64)
    assert got.potential.dtype == np.complex64 and got.gradient.dtype == np.complex64
    assert np.array_equal(got.potential, want.potential.astype(np.complex64))
    assert np.array_equal(got.gradient, want.gradient.astype(np.complex64))
    fmm.close()


@pytest.mark.parametrize("p", [10, 11])
def test_local_expansions_keep_their_precision(p):
    """A unit source at a leaf's centre, targets within 0.11 half-widths of the centres of leaves two
    and three away: one translation and L2P, cut off below 1e-16 of the potential at this k.  The
    error is rounding: 2.5e-16 rms with a sum per degree in L2P (2.3e-16 with three sums over the
    degrees), 3.5e-16 with one sum over all coefficients; the bound lies between."""
    rng = np.random.default_rng(2)
    c = (np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) / 4
    t = np.repeat(c, 100, axis=0) + np.round((rng.random((6400, 3)) * 2 - 1) * 0.11 / 8 * 2 ** 20) / 2 ** 20
    x, k = np.full((1, 3), 0.125), 8.0
    b = F.FmmBuilder(p).gradients().max_points_per_leaf(150).precision("f64")
    plan = b.plan(x, t).plan_arrays()
    plan["lower"], plan["side"] = np.zeros(3), 1.0  # the leaves' centres exactly at the grid's
    fmm = b.upload(plan, x, t)
    assert fmm.info()["nleaves"] == 64
    phi = fmm.helmholtz_evaluate(k, np.ones((1, 1))).potential[0]
    far = np.floor(t * 4).max(axis=1) >= 2
    r = np.sqrt(((t - x).astype(np.longdouble) ** 2).sum(axis=1))
    scale = 4 * np.longdouble("3.14159265358979323846264") * r
    err = np.hypot(phi.real - np.cos(k * r) / scale, phi.imag - np.sin(k * r) / scale).astype(float)
    want = (1 / scale).astype(float)
    assert np.sqrt((err[far] ** 2).sum() / (want[far] ** 2).sum()) < 2.9e-16
    fmm.close()


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_handles_of_few_and_many_vectors_side_by_side(cloud, precision):
    """The leaf sums' shared memory grows with the vectors: a handle of one vector set up after one of
    many leaves the other's launches as they were."""
    x, q = cloud
    b = F.FmmBuilder(9).max_points_per_leaf(30).precision(precision)
    qs = np.stack([q * (v + 1.0) for v in range(12)], axis=1)
    many = b.vectors(12).build(x)
    want = many.helmholtz_evaluate(4.0, qs).potential
    one = b.vectors(1).build(x)
    one.helmholtz_evaluate(4.0, q)
    got = many.helmholtz_evaluate(4.0, qs).potential
    assert np.array_equal(got, want)
    one.close()
    many.close()
