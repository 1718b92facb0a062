"""The f64 near field: items of every slot count (a leaf's remainders), flushes of exactly 64
sources and one more, near rows of more entries than a warp has lanes, one to five
charge vectors, coincident points, against direct sums; the complex (Helmholtz) form too."""
import numpy as np
import pytest

import fmm_b200 as F

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b)))


def direct(x, t, q, k=0.0):
    d = t[:, None, :] - x[None, :, :]
    r = np.sqrt((d * d).sum(-1))
    with np.errstate(divide="ignore", invalid="ignore"):
        inv = np.where(r > 0, 1.0 / r, 0.0)
    g = np.exp(1j * k * r) * inv if k else inv
    rad = g * (1j * k * r - 1.0) * inv * inv if k else -inv ** 3
    f = 1.0 / (4.0 * np.pi)
    return f * (g @ q).T, f * np.einsum("ij,ijk,jv->vik", rad, d, q)


# a tree of one leaf: the evaluation is the near field alone.  1e-13: f64 sums of at most 200
# terms that cancel (measured 1e-15)
@pytest.mark.parametrize("m", [1, 2, 3, 5])
def test_one_leaf_is_the_direct_sum(m):
    rng = np.random.default_rng(m)
    for nt in (1, 2, 4, 5, 8, 9, 16, 17, 24, 25, 32, 33, 57):
        ns = int(rng.choice([1, 3, 31, 63, 64, 65, 128, 130]))
        x, t = rng.random((ns, 3)), rng.random((nt, 3))
        t[: min(nt, ns) // 2] = x[: min(nt, ns) // 2]  # coincident pairs are left out
        q = rng.standard_normal((ns, m))
        if ns == 1 and nt >= 1:
            t[0] = t[0] + 0.25
        fmm = F.FmmBuilder(3).gradients().vectors(m).max_points_per_leaf(200).build(x, t)
        out = fmm.evaluate(q)
        phi, g = direct(x, t, q)
        assert rel(out.potential, phi) < 1e-13 and rel(out.gradient, g) < 1e-13, (ns, nt)
        z = q + 1j * rng.standard_normal((ns, m))
        hz = fmm.helmholtz_near(3.0, z)
        phi, g = direct(x, t, z, 3.0)
        assert rel(hz.potential, phi) < 1e-13 and rel(hz.gradient, g) < 1e-13, (ns, nt)
        fmm.close()


# 1e-12: the f64 path's bound against the oracle on the same tree and order
def test_long_near_rows_match_oracle(oracle):
    rng = np.random.default_rng(11)
    x = np.concatenate([rng.random((300, 3)), 0.5 + 1e-3 * rng.random((6000, 3))])  # one dense corner
    q = rng.standard_normal(len(x))
    fmm = F.FmmBuilder(5).gradients().max_points_per_leaf(4).build(x)
    arrays = fmm.plan_arrays()
    assert np.diff(arrays["near_rows"]).max() > 32
    out = fmm.evaluate(q)
    phi, g = oracle.fmm(x, q, x, 5, 4, gradients=True, threads=8)
    assert rel(out.potential, phi) < 1e-12 and rel(out.gradient, g) < 1e-12
    fmm.close()


# phases below a quarter turn, over many turns, beyond 1e5 (the library's reduction) and damped.
# 1e-13 as above plus the phase's own rounding: k r with k, r each rounded, so up to a few
# 2^-53 k r of a turn's angle (r below 2 in these boxes)
@pytest.mark.parametrize("k", [0.5, 40.0, 700.0, 4e5, 3.0 + 2.0j])
def test_helmholtz_phases(k):
    rng = np.random.default_rng(5)
    x, t = rng.random((130, 3)), rng.random((57, 3))
    z = rng.standard_normal((130, 1)) + 1j * rng.standard_normal((130, 1))
    fmm = F.FmmBuilder(3).gradients().max_points_per_leaf(200).build(x, t)
    out = fmm.helmholtz_near(k, z)
    phi, g = direct(x, t, z, k)
    tol = 1e-13 + 8 * 2.0 ** -53 * abs(k) * 2
    assert rel(out.potential, phi) < tol and rel(out.gradient, g) < tol
    fmm.close()


# a growing wave (Im k < 0) at source counts on and off the flush size.  In the leaf's half-widths
# Im k is down to -20: every pair is finite (at most e^(20 sqrt 3)), a point 1,000 half-widths
# away would not be.  1e-13 as above plus the rounding of the exponent and the phase (|k| r, r below 2)
@pytest.mark.parametrize("k", [3.0 - 1.0j, -2.0j, 5.0 - 40.0j])
@pytest.mark.parametrize("ns", [1, 2, 63, 64, 65, 130])
def test_growing_wave(k, ns):
    rng = np.random.default_rng(ns)
    x, t = rng.random((ns, 3)), rng.random((41, 3))
    z = rng.standard_normal((ns, 1)) + 1j * rng.standard_normal((ns, 1))
    fmm = F.FmmBuilder(3).gradients().max_points_per_leaf(200).build(x, t)
    assert fmm.info()["nleaves"] == 1
    out = fmm.helmholtz_near(k, z)
    phi, g = direct(x, t, z, k)
    tol = 1e-13 + 8 * 2.0 ** -53 * abs(k) * 2
    assert rel(out.potential, phi) < tol and rel(out.gradient, g) < tol
    fmm.close()


# a source that coincides with a target is left out of its sums whatever the source's charge
@pytest.mark.parametrize("bad", [np.nan, np.inf, complex(1.0, -np.inf)])
@pytest.mark.parametrize("k", [2.0, 2.0 - 0.5j])
def test_a_coincident_charge_that_is_no_number_is_left_out(bad, k):
    rng = np.random.default_rng(9)
    x = rng.random((70, 3))
    z = rng.standard_normal((70, 1)) + 1j * rng.standard_normal((70, 1))
    z[13] = bad
    fmm = F.FmmBuilder(3).gradients().max_points_per_leaf(200).build(x)
    out = fmm.helmholtz_near(k, z)
    rest = np.arange(70) != 13
    phi, g = direct(x[rest], x[13:14], z[rest], k)
    assert rel(out.potential[:, 13:14], phi) < 1e-13 and rel(out.gradient[:, 13:14], g) < 1e-13
    assert not np.isfinite(out.potential[:, rest]).any()
    fmm.close()


def one_pair(t):
    """Points on a grid of 2^-20 and one source at (2^-20, 2^-20, 2^-20), in one leaf of half-width
    1/2 at (1/2, 1/2, 1/2): the leaf's coordinates, the pairs' differences and r^2 are exact."""
    x = np.full((1, 3), 2.0 ** -20)
    b = F.FmmBuilder(3).gradients().max_points_per_leaf(1 << 20)
    plan = b.plan(x, t).plan_arrays()
    plan["lower"], plan["side"] = np.zeros(3), 1.0
    d = 2.0 * (t - x)
    return b.upload(plan, x, t), d, (d * d).sum(-1)


SCALE = 4.0 * 3.141592653589793 * 0.5  # the kernels' output scale of this leaf, the same double


# The term of the gradient, q / r^3 d / (4 pi r_t^2) at k = 0: 1/r^3 to 6.6e-17 rms (a division by
# r2 r has 8.2e-17); with the product's and the output scale's roundings (4.7e-17 each) 9.4e-17
def test_helmholtz_gradient_term_keeps_the_precision_of_a_division():
    rng = np.random.default_rng(3)
    t = rng.integers(2, 1 << 20, (20000, 3)) / 2.0 ** 20
    fmm, d, r2 = one_pair(t)
    out = fmm.helmholtz_near(0.0, np.ones((1, 1)))
    want = -d / (np.sqrt(r2.astype(np.longdouble)) * r2)[:, None] / np.longdouble(SCALE * 0.5)
    err = ((out.gradient[0].real - want) / want).astype(float)
    assert np.sqrt((err * err).mean()) < 1.0e-16
    fmm.close()


# 1/r against the rounded value: 0.51 ulp, as rsqrt(), so that all but about one value in a hundred
# (those within 0.01 ulp of a midpoint) are the rounded value's floats
def test_inverse_distance_is_rounded_as_rsqrt():
    rng = np.random.default_rng(4)
    t = rng.integers(2, 1 << 20, (200000, 3)) / 2.0 ** 20
    fmm, d, r2 = one_pair(t)
    phi = fmm.evaluate(np.ones(1)).potential[0]
    y = 1 / np.sqrt(r2.astype(np.longdouble))
    assert (phi != y.astype(float) / SCALE).mean() < 0.01
    err = ((phi * np.longdouble(SCALE) - y) / y).astype(float)
    assert np.abs(err).max() < (0.51 + 0.5) * 2.0 ** -52  # and the scale's division
    fmm.close()


# Sine and cosine of phases k r, k and r exact, over [0, 1e5] and beyond (the library's): 3.2e-17 rms
# and 1.25e-16 at most off, as sincos().  The potential rounds three times more (1/r, the product, the
# output scale: 2^-53 each at most), so against the same chain from rounded cosines, whose own error
# is 2.6e-17 rms, the rms may grow by sqrt((3.2^2 + 33) / (2.6^2 + 33)) = 1.04
@pytest.mark.parametrize("k", [1.0, 37.0, 2000.0, 1e5, 4e6])
def test_sine_and_cosine_are_as_good_as_sincos(k):
    rng = np.random.default_rng(6)
    t = np.full((50000, 3), 2.0 ** -20)
    t[:, 0] = rng.integers(2, 1 << 20, 50000) / 2.0 ** 20
    fmm, d, r2 = one_pair(t)
    r = d[:, 0]
    phase = (k * 0.5 * r).astype(np.longdouble)
    phi = fmm.helmholtz_near(k, np.ones((1, 1))).potential[0]
    for got, want in ((phi.real, np.cos(phase)), (phi.imag, np.sin(phase))):
        err = (got * np.longdouble(SCALE) * r - want).astype(float)
        best = (want.astype(float) * (1 / r) / SCALE * np.longdouble(SCALE) * r - want).astype(float)
        assert np.sqrt((err * err).mean()) < 1.1 * np.sqrt((best * best).mean())
        assert np.abs(err).max() < 1.25e-16 + 3 * 2.0 ** -53
    fmm.close()
