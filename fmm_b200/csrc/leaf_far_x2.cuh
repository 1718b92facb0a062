// L2P and M2P, and the harmonic rows they and P2M / P2L take, each complex harmonic one pair
// (re, im): in f32 on the packed f32x2 pipe of sm_100 (FFMA2 / FADD2 / FMUL2), in f64 the same
// code on pairs of doubles.  The gradients' sums are those of the ladder identities
//   (d/dx - i d/dy) phi = sum L_{k+1}^{mu+1} R_k^mu - conj(sum L_{k+1}^{mu-1} R_k^mu)
//   d/dz phi = sum w_mu Re(L_{k+1}^mu R_k^mu)          (M2P: M_{k-1} and I_k, sign -)
// taken coefficient by coefficient: a coefficient c = (a, b) of degree n and order mu adds
//   potential        w Re(c H)            H the harmonic of (n, mu)
//   d/dz             w Re(c W)            W the harmonic of (n -+ 1, mu)      (M2P: minus)
//   d/dx - i d/dy    c U - conj(c V)      U, V the harmonics of (n -+ 1, mu -+ 1)
// with w = 1 for mu = 0 and 2 otherwise, L2P taking the row below (n - 1) and M2P the row
// above (n + 1).  With S = U - V and T = U + V,
//   Re(c U - conj(c V)) = a S.re - b S.im,   Im(c U - conj(c V)) = a T.im + b T.re,
// so a coefficient is read once and costs four packed fused multiply-adds ((a, b) times H, W
// and S, (b, a) times T, into pair sums whose real and imaginary products are summed apart)
// and S, T two packed adds.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "harmonics.cuh"

namespace fmmb {

// pairs of T and their packed operations
template <typename T>
struct Pair2;
template <>
struct Pair2<float> {
    using type = float2;
};
template <>
struct Pair2<double> {
    using type = double2;
};
__device__ __forceinline__ float2 mk2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 mk2(double a, double b) { return make_double2(a, b); }
template <typename T>
__device__ __forceinline__ typename Pair2<T>::type x2(T a) {
    return mk2(a, a);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float fma1(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 mul2(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double2 add2(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double fma1(double a, double b, double c) { return fma(a, b, c); }

// The row recursions of the solid harmonics (fmm-math/src/harmonics.rs:118-187) with both parts of a
// harmonic in one packed instruction and the recursion's constants folded at compile
// time (a multiplication by 1 / ((n + m)(n - m)), no division): step(n) forms row n into
// c (m = 0..n), keeping rows n - 1 (pr) and n - 2 (pp); rows in order n = 0, 1, 2, ...
template <int PMAX, typename T = float>
struct RegularRows2 {
    using T2 = typename Pair2<T>::type;
    T x, y, z;
    T2 nr2;
    T2 pp[PMAX + 2], pr[PMAX + 2], c[PMAX + 2];  // one spare slot
    __device__ __forceinline__ void init(T x_, T y_, T z_) {
        x = x_;
        y = y_;
        z = z_;
        nr2 = x2(-(x * x + y * y + z * z));
    }
    __device__ __forceinline__ void step(int n) {
#pragma unroll
        for (int m = 0; m < n; ++m) {
            pp[m] = pr[m];
            pr[m] = c[m];
        }
        if (n == 0) {
            c[0] = mk2(T(1), T(0));
            return;
        }
        const T2 zn = x2(T(2 * n - 1) * z);
#pragma unroll
        for (int m = 0; m <= n; ++m) {
            if (m + 2 <= n) {
                // R_n^m = ((2n - 1) z R_{n-1}^m - r^2 R_{n-2}^m) / ((n + m)(n - m))
                const T inv_den = T(1) / T((n + m) * (n - m));
                c[m] = mul2(x2(inv_den), fma2(zn, pr[m], mul2(nr2, pp[m])));
            } else if (m + 1 == n) {
                c[m] = mul2(x2(z), pr[m]);
            } else {
                const T sc = T(1) / T(2 * n);
                const T a = pr[n - 1].x, b = pr[n - 1].y;
                c[m] = mk2((x * a - y * b) * sc, (x * b + y * a) * sc);
            }
        }
    }
};

template <int PMAX, typename T = float>
struct IrregularRows2 {
    using T2 = typename Pair2<T>::type;
    T x, y, z, inv_r, inv_r2;
    T2 ir2;
    T2 pp[PMAX + 2], pr[PMAX + 2], c[PMAX + 2];
    __device__ __forceinline__ void init(T x_, T y_, T z_, T inv_r_) {
        x = x_;
        y = y_;
        z = z_;
        inv_r = inv_r_;
        inv_r2 = inv_r * inv_r;
        ir2 = x2(inv_r2);
    }
    __device__ __forceinline__ void step(int n) {
#pragma unroll
        for (int m = 0; m < n; ++m) {
            pp[m] = pr[m];
            pr[m] = c[m];
        }
        if (n == 0) {
            c[0] = mk2(inv_r, T(0));
            return;
        }
        // I_n^m = ((2n - 1) z I_{n-1}^m - (n - 1 - m)(n - 1 + m) I_{n-2}^m) / r^2
        const T2 zn = x2(T(2 * n - 1) * z);
#pragma unroll
        for (int m = 0; m <= n; ++m) {
            if (m + 2 <= n) {
                const T2 k2 = x2(-T((n - 1 - m) * (n - 1 + m)));
                c[m] = mul2(ir2, fma2(zn, pr[m], mul2(k2, pp[m])));
            } else if (m + 1 == n) {
                c[m] = mul2(ir2, mul2(zn, pr[m]));
            } else {
                const T sc = T(2 * n - 1) * inv_r2;
                const T a = pr[n - 1].x, b = pr[n - 1].y;
                c[m] = mk2((x * a - y * b) * sc, (x * b + y * a) * sc);
            }
        }
    }
};

// The sums of one evaluation; the orders mu > 0 weighted 2 at the end.
template <typename T>
struct LadderSums {
    using T2 = typename Pair2<T>::type;
    T f0 = T(0), d0 = T(0), gxs = T(0), gys = T(0);  // mu = 0 (b = 0, H and W real)
    T2 f1 = mk2(T(0), T(0)), d1 = mk2(T(0), T(0));
    T2 sa = mk2(T(0), T(0)), tb = mk2(T(0), T(0));

    // coefficient (a, b) of order mu with harmonics H (potential), W (d/dz) and U, V (the
    // ladder); HAS_*: that harmonic exists for this coefficient
    template <bool MU0, bool HAS_W, bool HAS_U, bool HAS_V>
    __device__ __forceinline__ void add(T a, T b, T2 H, T2 W, T2 U, T2 V) {
        T2 D = mk2(T(0), T(0)), A = mk2(T(0), T(0));  // S, T
        if (HAS_U && HAS_V) {
            D = fma2(V, x2(T(-1)), U);
            A = add2(U, V);
        } else if (HAS_U) {
            D = U;
            A = U;
        } else if (HAS_V) {
            D = mk2(-V.x, -V.y);
            A = V;
        }
        if (MU0) {
            f0 = fma1(a, H.x, f0);
            if (HAS_W) d0 = fma1(a, W.x, d0);
            if (HAS_U || HAS_V) {
                gxs = fma1(a, D.x, gxs);
                gys = fma1(a, A.y, gys);
            }
        } else {
            const T2 ab = mk2(a, b);
            f1 = fma2(ab, H, f1);
            if (HAS_W) d1 = fma2(ab, W, d1);
            if (HAS_U || HAS_V) {
                sa = fma2(ab, D, sa);
                tb = fma2(mk2(b, a), A, tb);
            }
        }
    }
    __device__ __forceinline__ void finish(T dz_sign, T& phi, T& gx, T& gy, T& gz) const {
        phi = f0 + T(2) * (f1.x - f1.y);
        gz = dz_sign * (d0 + T(2) * (d1.x - d1.y));
        gx = gxs + (sa.x - sa.y);
        gy = -(gys + (tb.x + tb.y));
    }
};

// f(n) for the rows n = I..E.  In f64 n is a compile-time constant, so that the rows are unrolled
// whatever their size: #pragma unroll gave up on them from p = 7 on, and they went through local
// memory (41,017 targets x 4 vectors at p = 10: the evaluation 1.47 -> 1.24 ms).
template <typename T, int I, int E, class F>
__device__ __forceinline__ void for_rows(F&& f) {
    if constexpr (sizeof(T) == 8) {
        if constexpr (I <= E) {
            f(std::integral_constant<int, I>{});
            for_rows<T, I + 1, E>(f);
        }
    } else {
#pragma unroll
        for (int n = I; n <= E; ++n) f(n);
    }
}

// L2P with gradients at (x, y, z) in the box's unit frame; L the local (real storage)
template <int P, typename T>
__device__ __forceinline__ void l2p_x2(const T* __restrict__ L, T x, T y, T z, T& phi, T& gx, T& gy, T& gz) {
    using T2 = typename Pair2<T>::type;
    const T2 zero = mk2(T(0), T(0));
    RegularRows2<P, T> h;
    h.init(x, y, z);
    LadderSums<T> s;
    for_rows<T, 0, P>([&](auto row) {
        const int n = row;
        h.step(n);
        // the coefficients of degree n: H = R_n^mu, W = R_{n-1}^mu, U = R_{n-1}^{mu-1},
        // V = R_{n-1}^{mu+1}
#pragma unroll
        for (int mu = 0; mu <= n; ++mu) {
            const T a = L[slot(n, mu)], b = mu ? L[slot(n, -mu)] : T(0);
            const T2 W = mu <= n - 1 ? h.pr[mu] : zero;
            const T2 U = mu >= 1 ? h.pr[mu >= 1 ? mu - 1 : 0] : zero;
            const T2 V = mu + 1 <= n - 1 ? h.pr[mu + 1] : zero;
            if (mu == 0) {
                if (n >= 2)
                    s.template add<true, true, false, true>(a, b, h.c[0], W, U, V);
                else if (n == 1)
                    s.template add<true, true, false, false>(a, b, h.c[0], W, U, V);
                else
                    s.template add<true, false, false, false>(a, b, h.c[0], W, U, V);
            } else if (mu + 1 <= n - 1) {
                s.template add<false, true, true, true>(a, b, h.c[mu], W, U, V);
            } else if (mu <= n - 1) {
                s.template add<false, true, true, false>(a, b, h.c[mu], W, U, V);
            } else {
                s.template add<false, false, true, false>(a, b, h.c[mu], W, U, V);
            }
        }
    });
    s.finish(T(1), phi, gx, gy, gz);
}

// M2P with gradients at (x, y, z) in the source box's unit frame; M the multipole
template <int P, typename T>
__device__ __forceinline__ void m2p_x2(const T* __restrict__ M, T x, T y, T z, T& phi, T& gx, T& gy, T& gz) {
    using T2 = typename Pair2<T>::type;
    constexpr int K = P + 1;
    const T2 zero = mk2(T(0), T(0));
    IrregularRows2<K, T> h;
    h.init(x, y, z, T(1) / sqrt(x * x + y * y + z * z));
    LadderSums<T> s;
    for_rows<T, 0, K>([&](auto row) {
        const int n = row;
        h.step(n);
        if (n == 0) return;
        // the coefficients of degree d = n - 1: H = I_d^mu, W = I_n^mu, U = I_n^{mu-1},
        // V = I_n^{mu+1}
        const int d = n - 1;
#pragma unroll
        for (int mu = 0; mu <= d; ++mu) {
            const T a = M[slot(d, mu)], b = mu ? M[slot(d, -mu)] : T(0);
            if (mu == 0)
                s.template add<true, true, false, true>(a, b, h.pr[0], h.c[0], zero, h.c[1]);
            else
                s.template add<false, true, true, true>(a, b, h.pr[mu], h.c[mu], h.c[mu - 1], h.c[mu + 1]);
        }
    });
    s.finish(T(-1), phi, gx, gy, gz);
}

// The potential alone of one expansion (f64)
template <int P, class Rows>
__device__ __forceinline__ double phi_eval(Rows& h, const double* __restrict__ E) {
    double f0 = 0.0;
    double2 f1 = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k <= P; ++k) {
        h.step(k);
        f0 = fma(E[slot(k, 0)], h.c[0].x, f0);
#pragma unroll
        for (int mu = 1; mu <= k; ++mu) f1 = fma2(make_double2(E[slot(k, mu)], E[slot(k, -mu)]), h.c[mu], f1);
    }
    return f0 + 2.0 * (f1.x - f1.y);
}

}  // namespace fmmb
