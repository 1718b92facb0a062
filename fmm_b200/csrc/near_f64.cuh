// The f64 near field (P2P) and output pass: Laplace 1/(4 pi r) and Helmholtz e^{ikr}/(4 pi r),
// potential and gradient.
//
// What bounds it: the FP64 pipe (64 lanes an SM).  A Laplace pair with its gradient takes 18
// of its instructions: 3 differences, 3 for r2, 5 for 1/r, 7 for the sums.
//
// Work split.  An item is up to 32 targets of one leaf in ns slots (a power of two); its
// K = 32 / ns lanes a target share the sources, so a leaf's remainder of 5 targets keeps
// 40 lanes' worth of work on 32 lanes instead of 5 (leaves hold about 24 targets on average:
// a lane a target left a quarter to a half of the lanes idle).  The near row's sources, taken
// as one run over its leaves, go through shared memory in flushes of 64, mapped to the target
// leaf's frame as y = fma(r, u, c) (the leaf itself unchanged); each flush's partial sums are
// added to the lane's totals in flush order, and the K lanes of a target are added by a fixed
// tree at the end.  With few items the flushes are dealt to W warps of a block and their
// partials added in flush order all the same, so a target's sums are the same floats whatever
// the number of items in the plan.
//
// Measured (gradients): 774.5 M near pairs of a cube of 1e6 points in 1.49 ms, 0.52 T pairs/s,
// against 2.04 ms for a lane a target with rsqrt(); whole evaluations, with the translations
// unchanged: a cube of 2,500 points 82 -> 44 us (8 warps an item), of 1e6 5.96 -> 5.39 ms;
// Helmholtz on 40,009 points 1.30 -> 0.78 ms.
//
// The rules of the reference's device kernels hold: d = u_t - y, r2 by explicit fma, and a
// pair is left out iff r2 == 0 (its 1/r is then 0).  The sum is added to the far-field partial
// and scaled once, phi = phi_hat/(4 pi r_t), g = g_hat/((4 pi r_t) r_t)
// (fmm-exec/src/fmm.rs:4750-4778), in caller order.
#pragma once

#include "helmholtz.cuh"
#include "kernels.cuh"

namespace fmmb {

// y[u] = 1 / sqrt(r2[u]), 0 at r2 == 0, for U independent pairs.  The hardware's estimate of the high word has 21 significant
// bits, so its square is exact and e = 1 - r2 y^2 takes one rounding; a third-order step
// (Householder's, y (1 + e/2 + 3 e^2 / 8)) then leaves e^3 5/16 < 2^-57 beside the last
// fma's rounding: at most 0.51 ulp (0.289 rms) measured, as rsqrt(), at five instructions instead
// of its slow-path tests.  Below 2^-1007 (and at 0) the library's form, behind one branch for the
// U pairs: a branch a pair kept the pairs' dependent chains from overlapping (the FP64 pipe was
// 39 % busy, the warps waiting on their own results).
// Returns whether any of them went that way (the only one in which r2 == 0 occurs).
template <int U>
__device__ __forceinline__ bool inv_dist(const double (&r2)[U], double (&y)[U]) {
    bool small = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        double a;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(a) : "d"(r2[u]));
        const double e = __fma_rn(-r2[u], a * a, 1.0);
        y[u] = __fma_rn(a * e, __fma_rn(0.375, e, 0.5), a);
        small |= __double2hiint(r2[u]) < 0x01000000;
    }
    if (small)
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (__double2hiint(r2[u]) < 0x01000000) y[u] = r2[u] == 0.0 ? 0.0 : rsqrt(r2[u]);
    return small;
}

// sin and cos of U phases.  Reduced to [-pi/4, pi/4] by Cody and Waite's two-step subtraction of
// n pi/2 (pi/2 as a double and the remainder, each step one fma), then the Taylor polynomials to
// x^17 and x^16, whose remainders there are below 2^-58; over [0, 1e5] at most 1.25e-16 off (3.2e-17
// rms), as sincos().
// Branch-free up to |x| = 1e5, so that the pairs' chains overlap; beyond it (and for infinities
// and NaN) the library's form.  Helmholtz on 40,009 points: 707 -> 682 us against sincos().
template <int U>
__device__ __forceinline__ void sin_cos(const double (&x)[U], double (&sn)[U], double (&cs)[U]) {
    bool far = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const double n = rint(x[u] * 0.63661977236758134);  // 2 / pi
        double r = __fma_rn(-n, 1.5707963267948966, x[u]);
        r = __fma_rn(-n, 6.123233995736766e-17, r);  // pi / 2 minus its double
        const double z = r * r;
        double s = 1.0 / 355687428096000.0, c = 1.0 / 20922789888000.0;  // 1 / 17!, 1 / 16!
        s = __fma_rn(s, z, -1.0 / 1307674368000.0);
        c = __fma_rn(c, z, -1.0 / 87178291200.0);
        s = __fma_rn(s, z, 1.0 / 6227020800.0);
        c = __fma_rn(c, z, 1.0 / 479001600.0);
        s = __fma_rn(s, z, -1.0 / 39916800.0);
        c = __fma_rn(c, z, -1.0 / 3628800.0);
        s = __fma_rn(s, z, 1.0 / 362880.0);
        c = __fma_rn(c, z, 1.0 / 40320.0);
        s = __fma_rn(s, z, -1.0 / 5040.0);
        c = __fma_rn(c, z, -1.0 / 720.0);
        s = __fma_rn(s, z, 1.0 / 120.0);
        c = __fma_rn(c, z, 1.0 / 24.0);
        s = __fma_rn(s, z, -1.0 / 6.0);
        c = __fma_rn(c, z, -0.5);
        s = __fma_rn(s * z, r, r);
        c = __fma_rn(c, z, 1.0);
        const int q = __double2int_rn(n);
        const double a = q & 1 ? c : s, b = q & 1 ? s : c;
        sn[u] = q & 2 ? -a : a;
        cs[u] = (q + 1) & 2 ? -b : b;
        far |= !(fabs(x[u]) <= 1e5);
    }
    if (far)
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (!(fabs(x[u]) <= 1e5)) sincos(x[u], &sn[u], &cs[u]);
}

// The Laplace pair of VB charge vectors (the geometry formed once).
template <bool GRAD_, int VB_>
struct NearLaplace {
    static constexpr bool GRAD = GRAD_, HELM = false;
    static constexpr int VB = VB_;
    static constexpr int Q = VB;                       // doubles of a source's charges
    static constexpr int C = VB * (GRAD ? 4 : 1);      // sums a target
    static constexpr int U = VB < 4 ? 4 : 2;           // pairs in flight a lane
    struct Const {};
    // U pairs, d[u] = u_t - y_u, q[u] the source's charges, added in order
    __device__ static __forceinline__ void pairs(const Const&, const double (&d)[U][3], const double (&q)[U][Q],
                                                 double (&a)[C]) {
        double r2[U], y[U];
#pragma unroll
        for (int u = 0; u < U; ++u) r2[u] = pair_r2<double>(d[u][0], d[u][1], d[u][2]);
        inv_dist<U>(r2, y);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const double y3 = GRAD ? y[u] * (y[u] * y[u]) : 0.0;
#pragma unroll
            for (int b = 0; b < VB; ++b) {
                double* s = a + b * (GRAD ? 4 : 1);
                s[0] = __fma_rn(q[u][b], y[u], s[0]);
                if (GRAD) {
                    const double w = -(q[u][b] * y3);
#pragma unroll
                    for (int k = 0; k < 3; ++k) s[1 + k] = __fma_rn(w, d[u][k], s[1 + k]);
                }
            }
        }
    }
};

// The Helmholtz pair (helmholtz.cuh's term): phi += q e / r, g += q ((damping - 1) + i phase)
// e d / r^3, e = exp(damping) (cos phase + i sin phase); 1/r and its powers from one inverse
// square root, r rounded from r2 / r with one correction step.
template <bool GRAD_>
struct NearHelmholtz {
    static constexpr bool GRAD = GRAD_, HELM = true;
    static constexpr int VB = 1;
    static constexpr int Q = 2;
    static constexpr int C = GRAD ? 8 : 2;
    static constexpr int U = 2;
    struct Const {
        double kre, kim;
    };
    __device__ static __forceinline__ void pairs(const Const& k, const double (&d)[U][3], const double (&qs)[U][Q],
                                                 double (&a)[C]) {
        double r2[U], y[U], q[U][Q];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            r2[u] = pair_r2<double>(d[u][0], d[u][1], d[u][2]);
            q[u][0] = qs[u][0];
            q[u][1] = qs[u][1];
        }
        if (inv_dist<U>(r2, y))
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (r2[u] == 0.0) q[u][0] = q[u][1] = 0.0;  // left out whatever its charge, infinite ones too
        double r[U], ph[U], sn[U], cs[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            r[u] = r2[u] * y[u];
            r[u] = __fma_rn(0.5 * y[u], __fma_rn(-r[u], r[u], r2[u]), r[u]);
            ph[u] = k.kre * r[u];
        }
        sin_cos<U>(ph, sn, cs);
        if (k.kim != 0.0)
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const double decay = exp(-(k.kim * r[u]));
                sn[u] *= decay;
                cs[u] *= decay;
            }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const double phase = ph[u], damping = -(k.kim * r[u]);
            const double qr = q[u][0] * cs[u] - q[u][1] * sn[u], qi = q[u][0] * sn[u] + q[u][1] * cs[u];  // q e
            a[0] = __fma_rn(qr, y[u], a[0]);
            a[1] = __fma_rn(qi, y[u], a[1]);
            if (GRAD) {
                // 1/r^3 = y^3 (1 + 3/2 (1 - r2 y^2)) = y h + y/2 (3 h (1 - r2 h) - l) for y^2 = h + l:
                // 0.41 ulp rms, where the division 1 / (r2 r) has 0.55 (and one rounding less after
                // it) and y * (y * y) 1.01
                const double h = y[u] * y[u], l = __fma_rn(y[u], y[u], -h);
                const double c3 = __fma_rn(3.0, h * __fma_rn(-r2[u], h, 1.0), -l);
                const double y3 = __fma_rn(0.5 * y[u], c3, y[u] * h), f = damping - 1.0;
                const double gr = (qr * f - qi * phase) * y3, gi = (qr * phase + qi * f) * y3;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    a[2 + 2 * c] = __fma_rn(gr, d[u][c], a[2 + 2 * c]);
                    a[3 + 2 * c] = __fma_rn(gi, d[u][c], a[3 + 2 * c]);
                }
            }
        }
    }
};

// Where the sums go.  Laplace: mode 0 adds the far partial and writes the scaled output in
// caller order, 1 adds into the leaf-order store (level calls), 2 writes the near field alone
// in leaf order; far_phi [v][t], far_g [v][t][3].  Helmholtz: mode 0 with complex far partials
// (null: none), [v][t][2] and [v][t][6].
struct NearArgs {
    DevPlan plan;
    P2pItems items;
    int m, near, mode;
    const double4* spos;
    const double* sq;  // [v][point] (Helmholtz: complex)
    const double4* tpos;
    double *far_phi, *far_g, *out_phi, *out_g;
    double k_re, k_im;  // the physical wavenumber
    int num_sms;        // of the device
};

constexpr int kNearFlush = 64;    // sources a flush
constexpr int kNearRecs = 64;     // near entries held at once
constexpr int kNearWarps = 4;     // warps (items) a block when items are not shared

template <class PK>
constexpr int near_stage_doubles() {  // x, y, z, charges, in 16-byte pairs
    return (3 + PK::Q + 1) / 2 * 2;
}

// Blocks an SM of the warp-an-item form with one vector: five (20 warps, 102 registers), since
// a pair's dependent chain and not the FP64 pipe bounds a warp: 1e6 points of a cube 1.49 ms
// against 1.73 with the 154 registers and 12 warps the compiler takes unasked (six blocks 1.50;
// two pairs in flight instead of four 1.58 to 1.61).
template <class PK>
constexpr int near_blocks(bool share) {
    return share || PK::VB > 1 ? 1 : PK::HELM ? 3 : 5;
}

// SHARE: the block's warps share one item (its flushes dealt round robin); else a warp an item.
template <class PK, bool SHARE>
__global__ void __launch_bounds__(SHARE ? 256 : 32 * kNearWarps, near_blocks<PK>(SHARE)) near_f64_kernel(NearArgs A) {
    constexpr int SD = near_stage_doubles<PK>(), C = PK::C;
    constexpr bool HELM = PK::HELM;
    constexpr int RW = SHARE ? 1 : kNearWarps;  // record sets a block
    static_assert(C * 32 <= kNearFlush * SD, "a warp's partial sums fit its stage");
    __shared__ double4 rec_frame[RW][kNearRecs];
    __shared__ int64_t rec_s0[RW][kNearRecs];
    __shared__ int rec_pre[RW][kNearRecs + 1];
    extern __shared__ __align__(16) double near_stage[];  // [warps][SD / 2][flush][2]
    const DevPlan& plan = A.plan;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = SHARE ? (int)(blockDim.x >> 5) : 1, ws = SHARE ? warp : 0, rw = SHARE ? 0 : warp;
    const int64_t item = SHARE ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * kNearWarps + warp;
    if (item >= A.items.count) return;
    double2* st = reinterpret_cast<double2*>(near_stage) + (size_t)warp * (SD / 2) * kNearFlush;
    const int leaf = A.items.leaf[item];
    const int box = plan.leaf_box[leaf];
    const int nn = A.items.n[item], ni = nn & 255, ns = nn >> 8;  // targets, slots (a power of two)
    const int ti = lane & (ns - 1), kk = lane / ns, K = 32 / ns;
    const int64_t t = A.items.t0[item] + (ti < ni ? ti : 0);
    const double4 tp = A.tpos[t];
    const int64_t n0 = plan.near_row[leaf], n1 = A.near ? plan.near_row[leaf + 1] : n0;
    const int64_t nt = plan.ntgt;
    const double rt = (plan.box_side ? plan.box_side[box] : plan.side) * pow2d(-(plan.level[box] + 1));
    const double phi_scale = 4.0 * 3.141592653589793 * rt;
    const double g_scale = phi_scale * rt;
    typename PK::Const kc;
    if constexpr (HELM) {
        kc.kre = A.k_re * rt;  // k_l = k r_l
        kc.kim = A.k_im * rt;
    }
    for (int v0 = 0; v0 < A.m; v0 += PK::VB) {
        const int nb = A.m - v0 < PK::VB ? A.m - v0 : PK::VB;
        double acc[C];
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] = 0.0;
        for (int64_t e0 = n0; e0 < n1; e0 += kNearRecs) {
            // the records of up to 64 near entries: frame, first source, sources before it
            const int ne = (int)(n1 - e0 < kNearRecs ? n1 - e0 : kNearRecs);
            if (!SHARE || ws == 0) {
                int cnt[2] = {0, 0};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int e = lane + 32 * h;
                    if (e >= ne) continue;
                    const int sl = plan.near_col[e0 + e];
                    double c[3] = {0.0, 0.0, 0.0}, r = 1.0;  // the leaf itself: y = fma(1, u, 0) = u
                    if (sl != leaf) rel_frame<double>(plan, plan.leaf_box[sl], box, c, r);
                    rec_frame[rw][e] = make_double4(c[0], c[1], c[2], r);
                    const int64_t s0 = plan.src_start[sl];
                    rec_s0[rw][e] = s0;
                    cnt[h] = (int)(plan.src_start[sl + 1] - s0);
                }
                int base = 0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    int x = cnt[h];
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x += y;
                    }
                    rec_pre[rw][lane + 32 * h] = base + x - cnt[h];
                    base += __shfl_sync(0xffffffffu, x, 31);
                }
                if (lane == 0) rec_pre[rw][kNearRecs] = base;
            }
            if (SHARE)
                __syncthreads();
            else
                __syncwarp();
            const int tot = rec_pre[rw][kNearRecs];
            const int nfl = (tot + kNearFlush - 1) / kNearFlush;
            // a lane's two sources of flush f, mapped; past the end: the last source without its charge
            // (a point of the run, so that a growing wave, Im k < 0, is finite there too)
            auto fetch = [&](int f, double (&s)[2][SD]) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int at = f * kNearFlush + lane + 32 * h, pos = at < tot ? at : tot - 1;
#pragma unroll
                    for (int c = 3; c < SD; ++c) s[h][c] = 0.0;
                    int lo = 0;  // the last entry starting at or before pos
#pragma unroll
                    for (int b = kNearRecs / 2; b; b >>= 1)
                        if (lo + b < ne && rec_pre[rw][lo + b] <= pos) lo += b;
                    const double4 fr = rec_frame[rw][lo];
                    const int64_t si = rec_s0[rw][lo] + (pos - rec_pre[rw][lo]);
                    const double4 u = A.spos[si];
                    s[h][0] = map_coord<double>(fr.w, u.x, fr.x);
                    s[h][1] = map_coord<double>(fr.w, u.y, fr.y);
                    s[h][2] = map_coord<double>(fr.w, u.z, fr.z);
                    if (at >= tot) continue;
                    if constexpr (HELM) {
                        const double2 q = reinterpret_cast<const double2*>(A.sq)[(int64_t)v0 * plan.nsrc + si];
                        s[h][3] = q.x;
                        s[h][4] = q.y;
                    } else {
#pragma unroll
                        for (int b = 0; b < PK::VB; ++b)
                            if (b < nb) s[h][3 + b] = A.sq[(int64_t)(v0 + b) * plan.nsrc + si];
                    }
                }
            };
            double nxt[2][SD];
            if (ws < nfl) fetch(ws, nxt);
            for (int f = ws; f - ws < nfl; f += W) {  // rounds of W flushes (every warp the same count)
                const bool have = f < nfl;
                double p[C];
#pragma unroll
                for (int c = 0; c < C; ++c) p[c] = 0.0;
                if (have) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int c = 0; c < SD / 2; ++c)
                            st[c * kNearFlush + lane + 32 * h] = make_double2(nxt[h][2 * c], nxt[h][2 * c + 1]);
                    __syncwarp();
                    if (f + W < nfl) fetch(f + W, nxt);  // in flight while this flush is summed
                    const int cnt = tot - f * kNearFlush < kNearFlush ? tot - f * kNearFlush : kNearFlush;
                    constexpr int U = PK::U;  // (a flush's padding keeps every group of U K inside it)
                    const int lim = (cnt + U * K - 1) / (U * K) * (U * K);
                    for (int s = kk; s < lim; s += U * K) {
                        double d[U][3], q[U][PK::Q];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            double w[SD];
#pragma unroll
                            for (int c = 0; c < SD / 2; ++c) {
                                const double2 x = st[c * kNearFlush + s + u * K];
                                w[2 * c] = x.x;
                                w[2 * c + 1] = x.y;
                            }
                            d[u][0] = sub_rn<double>(tp.x, w[0]);
                            d[u][1] = sub_rn<double>(tp.y, w[1]);
                            d[u][2] = sub_rn<double>(tp.z, w[2]);
#pragma unroll
                            for (int b = 0; b < PK::Q; ++b) q[u][b] = w[3 + b];
                        }
                        PK::pairs(kc, d, q, p);
                    }
                    __syncwarp();
                }
                if (SHARE) {
                    // the round's partials added in flush order
                    double* ps = reinterpret_cast<double*>(st);
                    if (have)
#pragma unroll
                        for (int c = 0; c < C; ++c) ps[c * 32 + lane] = p[c];
                    __syncthreads();
                    if (ws == 0) {
                        const int nw = nfl - f < W ? nfl - f : W;
                        for (int w = 0; w < nw; ++w)
#pragma unroll
                            for (int c = 0; c < C; ++c)
                                acc[c] += near_stage[(size_t)w * SD * kNearFlush + c * 32 + lane];
                    }
                    __syncthreads();
                } else {
#pragma unroll
                    for (int c = 0; c < C; ++c) acc[c] += p[c];
                }
            }
            if (SHARE)
                __syncthreads();  // the records are read
            else
                __syncwarp();
        }
        if (SHARE && ws != 0) continue;
        // the K lanes of a target
        for (int o = ns; o < 32; o <<= 1)
#pragma unroll
            for (int c = 0; c < C; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
        if (kk != 0 || ti >= ni) continue;
        if constexpr (HELM) {
            const int64_t at = (int64_t)v0 * nt + t;
            const int64_t i = (int64_t)v0 * nt + plan.tgt_perm[t];
            if (A.far_phi) {  // the far field's partials, added after the near sums
                acc[0] += A.far_phi[2 * at];
                acc[1] += A.far_phi[2 * at + 1];
                if (PK::GRAD)
#pragma unroll
                    for (int c = 0; c < 6; ++c) acc[2 + c] += A.far_g[6 * at + c];
            }
            A.out_phi[2 * i] = acc[0] / phi_scale;
            A.out_phi[2 * i + 1] = acc[1] / phi_scale;
            if (PK::GRAD)
#pragma unroll
                for (int c = 0; c < 6; ++c) A.out_g[6 * i + c] = acc[2 + c] / g_scale;
        } else {
#pragma unroll
            for (int b = 0; b < PK::VB; ++b) {
                if (b >= nb) break;
                const double* a = acc + b * (PK::GRAD ? 4 : 1);
                const int64_t at = (int64_t)(v0 + b) * nt + t;
                if (A.mode == 2) {
                    A.out_phi[at] = a[0];
                    if (PK::GRAD)
#pragma unroll
                        for (int k = 0; k < 3; ++k) A.out_g[3 * at + k] = a[1 + k];
                    continue;
                }
                const double ph = A.far_phi[at] + a[0];
                if (A.mode == 1) {
                    A.far_phi[at] = ph;
                    if (PK::GRAD)
#pragma unroll
                        for (int k = 0; k < 3; ++k) A.far_g[3 * at + k] += a[1 + k];
                    continue;
                }
                const int64_t i = (int64_t)(v0 + b) * nt + plan.tgt_perm[t];
                A.out_phi[i] = ph / phi_scale;
                if (PK::GRAD)
#pragma unroll
                    for (int k = 0; k < 3; ++k) A.out_g[3 * i + k] = (A.far_g[3 * at + k] + a[1 + k]) / g_scale;
            }
        }
    }
}

// launched from p2p_launch.cu (the kernels do not depend on the expansion order)
void launch_near_laplace_f64(const NearArgs& a, bool gradients, cudaStream_t s);
void launch_near_helmholtz_f64(const NearArgs& a, bool gradients, cudaStream_t s);

}  // namespace fmmb
