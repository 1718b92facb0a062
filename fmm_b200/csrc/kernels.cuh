// Device kernels of the FMM evaluation passes (one rank, one GPU).
//
// Data in HBM (all level-major, see plan.hpp):
//   multipoles / locals : [box][vector][(p+1)^2]            (T)
//   source points       : xyz as T4 (w unused) + charges [vector][point]  (leaf order)
//   target points       : xyz as T4                                       (leaf order)
//   far-field partials  : phi [vector][target], grad [vector][target][3]  (f64)
//   output              : caller order, phi [vector][target], grad [...][3] (f64)
// Every kernel adds into its output in a fixed order per output value, with no atomics,
// so two evaluations are bit-identical.
#pragma once

#include <cstdint>

#include "harmonics.cuh"
#include "leaf_far_x2.cuh"

namespace fmmb {

template <typename T>
struct Vec4;
template <>
struct Vec4<double> {
    using type = double4;
};
template <>
struct Vec4<float> {
    using type = float4;
};

struct DevPlan {
    int nlevels;
    double side;
    const int32_t* level;      // per box
    const uint32_t* idx;       // 3 per box
    const int32_t* parent;
    const int32_t* child_first;
    const int32_t* box_leaf;
    const int64_t* src_below;
    const int64_t* tgt_below;
    const int32_t* leaf_box;
    const int64_t* src_start;
    const int64_t* tgt_start;
    const int64_t* tgt_perm;
    const int64_t* src_perm;
    const int64_t *near_row, *w_row, *x_row, *v_row;
    const int32_t *near_col, *w_col, *x_col, *v_col, *v_off;
    int64_t nsrc, ntgt;
    const double* box_side;  // forests: the domain side of each box's tree (null: `side`)
};

// 2^e for |e| <= 126, built from the exponent field (exact, no library call)
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }
__device__ __forceinline__ double pow2d(int e) { return __longlong_as_double((long long)(1023 + e) << 52); }
template <typename T>
__device__ __forceinline__ T pow2(int e);
template <>
__device__ __forceinline__ float pow2<float>(int e) { return pow2f(e); }
template <>
__device__ __forceinline__ double pow2<double>(int e) { return pow2d(e); }

// relative frame of box s seen from box t (CONVENTIONS 3.13 "Relative frames"):
// c = (C_L(s) - C_L(t)) 2^(l_t - L), r = 2^(l_t - l_s); exact in f32 and f64 (the
// integer difference has at most 17 bits and the scale is a power of two).
template <typename T>
__device__ __forceinline__ void rel_frame(const DevPlan& P, int s, int t, T c[3], T& r) {
    int ls = P.level[s], lt = P.level[t];
    int L = ls > lt ? ls : lt;
    const T scale = pow2<T>(lt - L);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int Cs = (int)((2u * P.idx[3 * s + k] + 1u) << (L - ls));
        int Ct = (int)((2u * P.idx[3 * t + k] + 1u) << (L - lt));
        c[k] = (T)(Cs - Ct) * scale;
    }
    r = pow2<T>(lt - ls);
}

// ---------------------------------------------------------------------------------
// Charge load: caller-order charges (m per point, point-major) -> leaf order [v][i].
// ---------------------------------------------------------------------------------
// (m vectors of a pass; the caller's array holds `stride` charges per point, the pass's
// first at q_caller[0])
template <typename T>
__global__ void charge_load_kernel(const double* __restrict__ q_caller, const int64_t* __restrict__ perm,
                                   int64_t n, int m, int stride, T* __restrict__ q_leaf, double* __restrict__ q64) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int64_t c = perm[i];
    for (int v = 0; v < m; ++v) {
        double q = q_caller[c * stride + v];
        q_leaf[(int64_t)v * n + i] = (T)q;
        if (q64) q64[(int64_t)v * n + i] = q;  // the mixed form keeps f64 charges for its f64 pairs
    }
}

// ---------------------------------------------------------------------------------
// P2M (rows = leaves, the leaf's own sources, unit frame) and P2L (rows = boxes, the sources
// of the X-list leaves, frame (c(t|s), r(t|s))): one warp per row.
//   multipole: M_n^m = sum q conj R_n^m(u);  X sum: X_n^m = sum q conj I_n^m((u - c)/r)
// P2L writes its sums to an array of their own (Lx, a box's rows as in Lc), so that every
// level's P2L is one launch beside the upward pass; the downward pass adds them.
//
// The row's sources, taken as one run over its entries, go 32 at a time: each lane forms one
// source's harmonics (conj X, the slots of harmonics.cuh) into shared memory, then the lanes
// hold the slots lane, lane + 32, ... and add q S over the 32 sources, for VB charge vectors at
// a time, in registers: four sources in order, the eight fours of a chunk as a tree, the chunks
// in f64, which rounds no more than a source a lane and a butterfly over the lanes (f32, random
// signs, in units of 2^-24 of the terms' 2-norm, 32 / 600 sources: 1.04 / 1.11, the butterfly 1.10 /
// 1.69, one sum over all sources 1.72 / 7.33).  The harmonics are so formed once per source and VB
// vectors, and a run over the X entries fills the lanes where single leaves of 8 to 24 sources
// left most of them idle: a batch of 700,000 points with 16 vectors at p = 6 takes 0.14 ms for
// P2M and 0.53 for P2L (one sum over all sources: 0.09 and 0.44), against 0.40 and 1.50 with the
// harmonics formed again for each vector (in f64, whose shared-memory rows of 32 fell in one
// bank, P2M of 1e6 points at p = 8 takes 0.09 ms against 0.20).  A vector's sums are the same
// floats for any VB.
// A handle of one f32 vector keeps the register form below where it is the faster one.
// ---------------------------------------------------------------------------------
// A lane's partial sums of a chunk: slots lane, lane + 32, ... of VB vectors
template <typename T, int NCL, int VB>
struct ChunkSum {
    using T2 = typename Pair2<T>::type;
    T2 v[NCL][(VB + 1) / 2];
    __device__ __forceinline__ T at(int c, int b) const { return b & 1 ? v[c][b / 2].y : v[c][b / 2].x; }
    // this + o, or o (first)
    __device__ __forceinline__ void add(const ChunkSum& o, bool plus) {
#pragma unroll
        for (int c = 0; c < NCL; ++c)
#pragma unroll
            for (int b = 0; b < (VB + 1) / 2; ++b) v[c][b] = plus ? add2(v[c][b], o.v[c][b]) : o.v[c][b];
    }
    // sources j0 .. j0 + 3 in order from zero
    template <int NC, int SR>
    __device__ __forceinline__ void four(const T* S, const T* Q, int lane, int j0) {
#pragma unroll
        for (int c = 0; c < NCL; ++c)
#pragma unroll
            for (int b = 0; b < (VB + 1) / 2; ++b) v[c][b] = mk2(T(0), T(0));
#pragma unroll
        for (int j = j0; j < j0 + 4; ++j) {
            T s[NCL];
#pragma unroll
            for (int c = 0; c < NCL; ++c) s[c] = S[(lane + 32 * c < NC ? lane + 32 * c : 0) * SR + j];
            if constexpr (VB == 1) {
                const T q = Q[j];
#pragma unroll
                for (int c = 0; c < NCL; ++c) v[c][0].x = fma1(q, s[c], v[c][0].x);
            } else {
                const T2* q2 = reinterpret_cast<const T2*>(Q + j * VB);
#pragma unroll
                for (int b = 0; b < VB / 2; ++b) {
                    const T2 q = q2[b];
#pragma unroll
                    for (int c = 0; c < NCL; ++c) v[c][b] = fma2(q, x2(s[c]), v[c][b]);
                }
            }
        }
    }
};

// the most vectors a pass: as many as keep their partial sums in registers (700,000 points with 16
// vectors at p = 6, P2M and P2L: 8 vectors 0.14 and 0.53 ms, 4 0.14 and 0.61, two passes of 8 over one
// chunk's harmonics 0.17 and 0.58)
template <int P, typename T>
constexpr int expand_most() {
    return sizeof(T) == 4 ? (P <= 8 ? 8 : 4) : P <= 7 ? 4 : 2;
}
template <int P, typename T>
constexpr int expand_smem(int vb) {
    return (int)sizeof(T) * ((nc_of(P) * 33 + 3) / 4 * 4 + 32 * vb);
}
template <int P, typename T, bool IRREG, int VB>
__global__ void __launch_bounds__(32) expand_kernel(DevPlan plan, int64_t row_begin, int64_t row_end,
                                                    const int32_t* __restrict__ rows, int m,
                                                    const typename Vec4<T>::type* __restrict__ spos,
                                                    const T* __restrict__ sq, T* __restrict__ out) {
    using T4 = typename Vec4<T>::type;
    using T2 = typename Pair2<T>::type;
    constexpr int NC = nc_of(P), NCL = (NC + 31) / 32, SR = 33;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* S = reinterpret_cast<T*>(smem_raw);    // [NC][33]
    T* Q = S + (NC * SR + 3) / 4 * 4;         // [32][VB]
    __shared__ T4 ent_frame[IRREG ? 32 : 1];  // an entry's frame c and 1 / r
    __shared__ int64_t ent_s0[IRREG ? 32 : 1];
    __shared__ int ent_pre[IRREG ? 33 : 1];   // sources before it in the batch
    const int lane = threadIdx.x;
    const int64_t idx = row_begin + blockIdx.x;  // rows[idx] when a row list is given
    if (idx >= row_end) return;
    const int64_t row = rows ? rows[idx] : idx;
    const int box = IRREG ? (int)row : plan.leaf_box[row];
    const int64_t x0 = IRREG ? plan.x_row[row] : 0, x1 = IRREG ? plan.x_row[row + 1] : 1;
    // a leaf without sources keeps its zero multipole
    if (IRREG ? x0 == x1 : plan.src_start[row + 1] == plan.src_start[row]) return;
    for (int v0 = 0; v0 < m; v0 += VB) {
        const int nb = m - v0 < VB ? m - v0 : VB;
        double run[NCL][VB];  // the finished chunks
#pragma unroll
        for (int c = 0; c < NCL; ++c)
#pragma unroll
            for (int b = 0; b < VB; ++b) run[c][b] = 0.0;
        for (int64_t e0 = x0; e0 < x1; e0 += 32) {
            const int ne = x1 - e0 < 32 ? (int)(x1 - e0) : 32;
            int64_t first = 0;  // P2M: the leaf's first source
            int tot;
            if constexpr (IRREG) {
                __syncwarp();
                int cnt = 0;
                if (lane < ne) {
                    const int sl = plan.x_col[e0 + lane];
                    T c[3], r;
                    rel_frame<T>(plan, box, plan.leaf_box[sl], c, r);  // (c(t|s), r(t|s))
                    T4 f;
                    f.x = c[0];
                    f.y = c[1];
                    f.z = c[2];
                    f.w = T(1) / r;
                    ent_frame[lane] = f;
                    const int64_t s0 = plan.src_start[sl];
                    ent_s0[lane] = s0;
                    cnt = (int)(plan.src_start[sl + 1] - s0);
                }
                int sum = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += y;
                }
                ent_pre[lane] = sum - cnt;
                tot = __shfl_sync(0xffffffffu, sum, 31);
                __syncwarp();
            } else {
                first = plan.src_start[row];
                tot = (int)(plan.src_start[row + 1] - first);
            }
            for (int cb = 0; cb < tot; cb += 32) {
                // past the end: the last source, uncharged
                const int pos = cb + lane < tot ? cb + lane : tot - 1;
                int64_t si = first + pos;
                T4 f;
                if constexpr (IRREG) {
                    int lo = 0;  // the last entry starting at or before pos
#pragma unroll
                    for (int b = 16; b; b >>= 1)
                        if (lo + b < ne && ent_pre[lo + b] <= pos) lo += b;
                    f = ent_frame[lo];
                    si = ent_s0[lo] + (pos - ent_pre[lo]);
                }
                const T4 p4 = spos[si];
#pragma unroll
                for (int b = 0; b < VB; ++b)
                    Q[lane * VB + b] = b < nb && cb + lane < tot ? sq[(int64_t)(v0 + b) * plan.nsrc + si] : T(0);
                auto slots = [&](auto& h) {
#pragma unroll
                    for (int n = 0; n <= P; ++n) {
                        h.step(n);
#pragma unroll
                        for (int mm = 0; mm <= n; ++mm) {
                            S[slot(n, mm) * SR + lane] = h.c[mm].x;
                            if (mm) S[slot(n, -mm) * SR + lane] = -h.c[mm].y;
                        }
                    }
                };
                if constexpr (IRREG) {
                    const T x = (p4.x - f.x) * f.w, y = (p4.y - f.y) * f.w, z = (p4.z - f.z) * f.w;
                    IrregularRows2<P, T> h;
                    h.init(x, y, z, T(1) / sqrt(x * x + y * y + z * z));
                    slots(h);
                } else {
                    RegularRows2<P, T> h;
                    h.init(p4.x, p4.y, p4.z);
                    slots(h);
                }
                __syncwarp();
                const int cnt = tot - cb < 32 ? tot - cb : 32;
                ChunkSum<T, NCL, VB> all;
#pragma unroll 1
                for (int h = 0; h < cnt; h += 16) {
                    ChunkSum<T, NCL, VB> half;
#pragma unroll
                    for (int e = 0; e < 16; e += 8) {
                        if (h + e >= cnt) break;
                        ChunkSum<T, NCL, VB> a, b;
                        a.template four<NC, SR>(S, Q, lane, h + e);
                        b.template four<NC, SR>(S, Q, lane, h + e + 4);
                        a.add(b, true);
                        half.add(a, e != 0);
                    }
                    all.add(half, h != 0);
                }
#pragma unroll
                for (int c = 0; c < NCL; ++c)
#pragma unroll
                    for (int b = 0; b < VB; ++b) run[c][b] += (double)all.at(c, b);
                __syncwarp();
            }
        }
#pragma unroll
        for (int c = 0; c < NCL; ++c) {
            const int k = lane + 32 * c;
            if (k >= NC) break;
#pragma unroll
            for (int b = 0; b < VB; ++b)
                if (b < nb) out[((int64_t)box * m + v0 + b) * ms_of(P) + k] = (T)run[c][b];
        }
    }
}

// ---------------------------------------------------------------------------------
// P2M / P2L, f32 single-vector form: one warp per row; lane j takes source points
// j, j+32, ... of every entry and accumulates q conj(X) for all (p+1)^2 slots in
// registers; one butterfly reduce-scatter per row then leaves every lane with
// NCP/32 finished slots (NCP = slots padded to a multiple of 32).  The summation order
// is fixed (per-lane partial sums, then a fixed tree), so results are repeatable.  It serves
// handles of one vector: P2M to p = 10 (above, its (p+1)^2 sums exceed the register file: 0.19
// against 0.08 ms for 1e6 points at p = 11) and P2L to p = 10 (4e6 points of a sphere at p = 8
// 0.22 against 0.30 ms; at p = 11 0.20 against 0.16).
// ---------------------------------------------------------------------------------
// One X-list entry of the f32 P2L, fixed at build (x_record_kernel): the source leaf's
// frame seen from the target box, (c(t|s), r(t|s)) of rel_frame<float>, and its sources,
// so that an entry costs one load, issued while the entry before it is summed.
struct __align__(16) XRec {
    float4 frame;  // (c0, c1, c2, r)
    long long s0;  // the source leaf's first source (leaf order)
    int ns;        // its sources
    int pad;
};

// Build time: thread per X entry of the boxes of `rows` (x_row order).
static __global__ void x_record_kernel(DevPlan plan, const int32_t* __restrict__ rows, int64_t nrows,
                                       XRec* __restrict__ rec) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    const int box = rows[r];
    for (int64_t e = plan.x_row[box]; e < plan.x_row[box + 1]; ++e) {
        const int sleaf = plan.x_col[e];
        float c[3], fr;
        rel_frame<float>(plan, box, plan.leaf_box[sleaf], c, fr);
        XRec x;
        x.frame = make_float4(c[0], c[1], c[2], fr);
        x.s0 = plan.src_start[sleaf];
        x.ns = (int)(plan.src_start[sleaf + 1] - plan.src_start[sleaf]);
        x.pad = 0;
        rec[e] = x;
    }
}

template <int P, bool IRREG>
__global__ void __launch_bounds__(32) expand_bfly_kernel(DevPlan plan, int64_t row_begin, int64_t row_end,
                                                         const int32_t* __restrict__ rows,
                                                         const float4* __restrict__ spos,
                                                         const float* __restrict__ sq, float* __restrict__ out,
                                                         const XRec* __restrict__ xrec = nullptr) {
    constexpr int NC = nc_of(P);
    constexpr int NCP = ((NC + 31) / 32) * 32;
    const int lane = threadIdx.x;
    const int64_t idx = row_begin + blockIdx.x;  // rows[idx] when a row list is given
    if (idx >= row_end) return;
    const int64_t row = rows ? rows[idx] : idx;
    int box, nent;
    int64_t ent0;
    if (!IRREG) {
        // a leaf without sources keeps its zero multipole; the test reads the leaf's source
        // range, which needs no load of its box first (the box is read beside it)
        box = plan.leaf_box[row];
        nent = 1;
        ent0 = 0;
        if (plan.src_start[row + 1] == plan.src_start[row]) return;
    } else {
        box = (int)row;
        ent0 = plan.x_row[row];
        nent = (int)(plan.x_row[row + 1] - ent0);
        if (nent == 0) return;
    }
    float w[NCP];
#pragma unroll
    for (int c = 0; c < NCP; ++c) w[c] = 0.0f;
    // P2L: the entries' records, the next one loaded while the current one is summed
    XRec xn{};
    if (IRREG) xn = xrec[ent0];
    for (int e = 0; e < nent; ++e) {
        float fc[3] = {0.0f, 0.0f, 0.0f}, fr = 1.0f;  // (c(t|s), r(t|s))
        int64_t s0, s1;
        if (IRREG) {
            const XRec xr = xn;
            if (e + 1 < nent) xn = xrec[ent0 + e + 1];
            fc[0] = xr.frame.x;
            fc[1] = xr.frame.y;
            fc[2] = xr.frame.z;
            fr = xr.frame.w;
            s0 = xr.s0;
            s1 = s0 + xr.ns;
        } else {
            s0 = plan.src_start[row];
            s1 = plan.src_start[row + 1];
        }
        const float finv = 1.0f / fr;
        // the lane's next source is loaded before its current one is summed
        int64_t si = s0 + lane;
        float4 pn = make_float4(0.f, 0.f, 0.f, 0.f);
        float qn = 0.f;
        if (si < s1) {
            pn = spos[si];
            qn = sq[si];
        }
        for (; si < s1; si += 32) {
            const float4 p4 = pn;
            const float q = qn;
            if (si + 32 < s1) {
                pn = spos[si + 32];
                qn = sq[si + 32];
            }
            const float x = (p4.x - fc[0]) * finv, y = (p4.y - fc[1]) * finv, z = (p4.z - fc[2]) * finv;
            // conj(X) q into the slots: (w[slot(n, mm)], w[slot(n, -mm)]) += (q, -q) * X_n^mm,
            // one packed fused multiply-add an order mm > 0 (the rows on the packed pipe,
            // leaf_far_x2.cuh)
            const float2 qq = make_float2(q, -q);
            auto scatter = [&](int n, const float2* cr) {
#pragma unroll
                for (int mm = 0; mm <= n; ++mm) {
                    if (mm == 0) {
                        w[slot(n, 0)] = fmaf(q, cr[0].x, w[slot(n, 0)]);
                    } else {
                        const float2 acc = __ffma2_rn(qq, cr[mm], make_float2(w[slot(n, mm)], w[slot(n, -mm)]));
                        w[slot(n, mm)] = acc.x;
                        w[slot(n, -mm)] = acc.y;
                    }
                }
            };
            if (!IRREG) {
                RegularRows2<P> h;
                h.init(x, y, z);
#pragma unroll
                for (int n = 0; n <= P; ++n) {
                    h.step(n);
                    scatter(n, h.c);
                }
            } else {
                IrregularRows2<P> h;
                h.init(x, y, z, rsqrtf(x * x + y * y + z * z));
#pragma unroll
                for (int n = 0; n <= P; ++n) {
                    h.step(n);
                    scatter(n, h.c);
                }
            }
        }
    }
    // reduce-scatter: after the step with offset s a lane keeps the half of its slots
    // selected by its bit s and adds the partner's copy of that half
#pragma unroll
    for (int s = 16, len = NCP / 2; s >= 1; s >>= 1, len >>= 1) {
        const bool upper = lane & s;
#pragma unroll
        for (int i = 0; i < len; ++i) {
            const float send = upper ? w[i] : w[i + len];
            const float keep = upper ? w[i + len] : w[i];
            w[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
    int base = 0;
#pragma unroll
    for (int s = 16, len = NCP / 2; s >= 1; s >>= 1, len >>= 1)
        if (lane & s) base += len;
    float* o = out + (int64_t)box * ms_of(P);
#pragma unroll
    for (int i = 0; i < NCP / 32; ++i) {
        const int c = base + i;
        if (c < NC) o[c] = w[i];
    }
}

// ---------------------------------------------------------------------------------
// M2M and L2L run as batched GEMMs too (the 8 octant tables): M2M's product T_o M_c is
// written to row c of Yo and the reduce below adds a parent's children in the reference's
// order; L2L's product T_o L_parent(c) is added to the child's local (add_local).
// ---------------------------------------------------------------------------------

// b += a (the fused M2L's level call: its sums start from zero, the locals are added to them)
template <typename T>
__global__ void add_rows_kernel(int64_t n, const T* __restrict__ a, T* __restrict__ b) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) b[i] = a[i] + b[i];
}

// M2M reduce for the parents of one level: M_p = sum over octants o (in order) of the
// products of its children that hold a source.  Block per parent, its threads over the slots
// of all vectors (a block of one vector's slots took 25 us a level with 16 vectors).
template <int P, typename T>
__global__ void m2m_reduce_kernel(DevPlan plan, const int32_t* __restrict__ parents, int64_t n, int m,
                                  const T* __restrict__ Yo, T* __restrict__ M) {
    constexpr int NC = nc_of(P), YS = ys_of(P);
    const int64_t j = blockIdx.x;
    if (j >= n) return;
    const int p = parents[j];
    const int c0 = plan.child_first[p];
    for (int vi = threadIdx.x; vi < m * NC; vi += blockDim.x) {
        const int v = vi / NC, i = vi % NC;
        T s = T(0);
#pragma unroll
        for (int o = 0; o < 8; ++o)
            if (plan.src_below[c0 + o]) s += Yo[((int64_t)(c0 + o) * m + v) * YS + i];
        M[((int64_t)p * m + v) * ms_of(P) + i] = s;
    }
}

// A child's local in the downward pass: L = (T_o L_parent + S) + X, S its V sum (in L), X its
// P2L sum when its X list is not empty (fmm-plan/src/operator.rs:34-45: the three are added,
// here as whole sums).
// x: whether the box takes an X sum (x_of, once a row).
template <typename T>
__device__ __forceinline__ bool x_of(const DevPlan& plan, int64_t box, const T* Lx) {
    return Lx && plan.x_row[box + 1] > plan.x_row[box];
}
__device__ __forceinline__ void add_local(double* L, const double* Lx, bool x, double2 v) {
    const double2 u = __ldcg(reinterpret_cast<const double2*>(L));
    v.x += u.x;
    v.y += u.y;
    if (x) {
        v.x += Lx[0];
        v.y += Lx[1];
    }
    *reinterpret_cast<double2*>(L) = v;
}

// The V sums of boxes [b0, b1) with a target below them: S = the V row's products in
// offset-index order (the product of V entry e sits at row vpos[e] of Yv, its place in the
// M2L tile list), from zero.  The evaluation writes L = S for every level in one launch, since
// no V sum waits for a parent's local, and the L2L pass adds its products to them; the level
// calls add S into L (accumulate).  Boxes below xend add their P2L sum last: level 2's, which
// no L2L reaches, or the boxes of a P2L level call (with_v = 0).
// Block per box, thread per slot; sixteen loads in flight, added in order.
template <typename T>
__device__ __forceinline__ bool has_x(const DevPlan& plan, int64_t b, const T* Lx, int64_t xend) {
    return Lx && b < xend && plan.x_row[b + 1] > plan.x_row[b];
}
template <int P, typename T>
__global__ void local_reduce_kernel(DevPlan plan, int64_t b0, int64_t b1, int m, int with_v, int accumulate,
                                    const T* __restrict__ Yv, const int64_t* __restrict__ vpos, T* __restrict__ Lc,
                                    const T* __restrict__ Lx, int64_t xend) {
    constexpr int NC = nc_of(P), YS = ys_of(P);
    const int64_t b = b0 + blockIdx.x;
    if (b >= b1 || plan.tgt_below[b] == 0) return;
    const int64_t e0 = plan.v_row[b], e1 = with_v ? plan.v_row[b + 1] : e0;
    const bool with_x = has_x(plan, b, Lx, xend);
    for (int v = 0; v < m; ++v)
        for (int i = threadIdx.x; i < NC; i += blockDim.x) {
            T s = T(0);
            int64_t e = e0;
            for (; e + 16 <= e1; e += 16) {  // sixteen rows in flight, added in row order
                T y[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) y[j] = __ldcs(Yv + (vpos[e + j] * m + v) * YS + i);
#pragma unroll
                for (int j = 0; j < 16; ++j) s += y[j];
            }
            for (; e + 4 <= e1; e += 4) {
                T y[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) y[j] = __ldcs(Yv + (vpos[e + j] * m + v) * YS + i);
#pragma unroll
                for (int j = 0; j < 4; ++j) s += y[j];
            }
            for (; e < e1; ++e) s += __ldcs(Yv + (vpos[e] * m + v) * YS + i);
            const int64_t at = (b * m + v) * ms_of(P) + i;
            if (accumulate) s = Lc[at] + s;
            if (with_x) s += Lx[at];
            Lc[at] = s;
        }
}

// The same reduce for f32 expansions with 16-byte accesses: a warp per box (4 a block).
// A box's m rows (its m vectors) are m NQ consecutive quads in the locals and in
// each of its V entries' products (ys_of = ms_of = 4 NQ), so the lanes take quads f, f + 32,
// ... of that run: every lane busy for any m (m = 16 at p = 6: 208 quads, 7 passes), 13 of
// 32 when the lanes held one vector's quads.  Every coefficient adds the same terms in the
// same order as local_reduce_kernel, so the floats are that kernel's.  The last quad of a
// row is read with its padding, which is never written.  Four blocks an SM in the launch
// bound leave room for sixteen 16-byte rows in flight.
__device__ __forceinline__ void add4(float4& s, const float4 y) {
    s.x += y.x;
    s.y += y.y;
    s.z += y.z;
    s.w += y.w;
}

template <int P, bool ONE>  // ONE: m = 1 at compile time
__global__ void __launch_bounds__(128, 4) local_reduce4_kernel(DevPlan plan, int64_t b0, int64_t b1, int m_, int with_v,
                                                            int accumulate, const float* __restrict__ Yv,
                                                            const int64_t* __restrict__ vpos, float* __restrict__ Lc,
                                                            const float* __restrict__ Lx, int64_t xend) {
    constexpr int NC = nc_of(P), YS = ys_of(P), MS = ms_of(P), NQ = (NC + 3) / 4;
    static_assert(YS == MS && MS == 4 * NQ, "a box's m rows are m NQ consecutive quads");
    const int m = ONE ? 1 : m_;
    const int64_t b = b0 + (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (b >= b1 || plan.tgt_below[b] == 0) return;
    const int64_t e0 = plan.v_row[b], e1 = with_v ? plan.v_row[b + 1] : e0;
    const int F = m * NQ;  // the box's quads, all vectors
    const bool with_x = has_x(plan, b, Lx, xend);
    for (int f = threadIdx.x & 31; f < F; f += 32) {
        const int q = f % NQ;  // the quad within its vector's row
        float4* out = reinterpret_cast<float4*>(Lc + b * m * MS) + f;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        auto row = [&](int64_t e) { return __ldcs(reinterpret_cast<const float4*>(Yv + vpos[e] * m * YS) + f); };
        int64_t e = e0;
        for (; e + 16 <= e1; e += 16) {  // sixteen rows in flight, added in row order
            float4 y[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) y[j] = row(e + j);
#pragma unroll
            for (int j = 0; j < 16; ++j) add4(s, y[j]);
        }
        for (; e + 8 <= e1; e += 8) {
            float4 y[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = row(e + j);
#pragma unroll
            for (int j = 0; j < 8; ++j) add4(s, y[j]);
        }
        for (; e + 4 <= e1; e += 4) {
            float4 y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = row(e + j);
#pragma unroll
            for (int j = 0; j < 4; ++j) add4(s, y[j]);
        }
        for (; e < e1; ++e) add4(s, row(e));
        if (accumulate) {
            float4 l = *out;
            add4(l, s);
            s = l;
        }
        if (with_x) add4(s, reinterpret_cast<const float4*>(Lx + b * m * MS)[f]);
        if (4 * q + 3 < NC) {
            *out = s;
        } else {  // the last quad: its coefficients below NC only (NC - 4q of them, 1 to 3)
            float* o = reinterpret_cast<float*>(out);
            o[0] = s.x;
            if (4 * q + 1 < NC) o[1] = s.y;
            if (4 * q + 2 < NC) o[2] = s.z;
        }
    }
}

// ---------------------------------------------------------------------------------
// Dense translations as batched GEMM, SIMT form (f32: M2M and L2L of wide levels and the M2L path
// without tensor cores; f64: the complex form above p = 8): the V pairs of every level are
// grouped by offset index d (fmm-kernels/src/translate.rs:61-74 batches them the same
// way); a block takes a tile of up to 64 pairs of one offset, stages A_d (column-major,
// so row k of the staged array holds column k) and the tile's source multipoles in
// shared memory, and writes the products Y[e] = A_d M_s (e = the pair's position in
// the target's V row).  Each thread holds 4 pairs x 6 output slots in registers.
// ---------------------------------------------------------------------------------
constexpr int kGemmPairs = 64;

// one element global -> shared by an asynchronous copy; zero-filled when !valid (the source
// address is then not read)
template <typename T>
__device__ __forceinline__ void gemm_cp_async(T* smem, const T* gmem, bool valid) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t n = valid ? (uint32_t)sizeof(T) : 0u;
    if constexpr (sizeof(T) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(gmem), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(gmem), "r"(n) : "memory");
}

// Shared memory of the SIMT GEMM: the table (columns as rows, NCP wide) and the tile's
// source rows, KC input slots at a time.  KC = the matrix order (one staging) where both
// fit in 200 KB; at higher degree in f64 the input slots are staged in chunks of KC, the
// accumulators kept in registers across the chunks (the same order of additions).  CPLX:
// the Helmholtz form, a complex expansion as one real vector of 2 (p+1)^2 entries (the
// real plane, then the imaginary plane) and the table a real 2n x 2n matrix.
template <int P, typename T, bool CPLX = false>
struct GemmShape {
    static constexpr int NC = nc_of(P);
    static constexpr int NE = CPLX ? 2 * NC : NC;  // matrix order
    static constexpr int NCP = 96 > NE ? 96 : ((NE + 15) / 16) * 16;
    static constexpr int ROW_BYTES = (NCP + kGemmPairs) * (int)sizeof(T);
    static constexpr int KC_FIT = (200 * 1024) / ROW_BYTES;
    static constexpr int KC = KC_FIT < NE ? KC_FIT : NE;
    static constexpr int SMEM = KC * ROW_BYTES;
};

// Y[pair] = A_d X[source] for a tile of pairs of one matrix d (column-major NE x NE).
// Rows: a box holds MV = m (real) or 2m (CPLX: rows 2v and 2v + 1 the real and imaginary
// planes of vector v) expansion rows of ms_of(P) slots; a product holds MV rows of
// ys_of(P) slots.
// ADD: the L2L of a level, Y = the locals: the product is added to the child's row,
// (T L_parent + S) + X.  The vectors are dealt over blockIdx.y (a block a tile with 16 vectors
// in turn took 80 us for levels of 24 to 104 tiles).
template <int P, typename T, bool CPLX = false, bool ADD = false>
__global__ void __launch_bounds__(256) m2l_gemm_kernel(const int32_t* __restrict__ tile_d,
                                                       const int64_t* __restrict__ tile_begin,
                                                       const int32_t* __restrict__ tile_count,
                                                       const int64_t* __restrict__ pair_e,
                                                       const int32_t* __restrict__ pair_src, int m,
                                                       const T* __restrict__ tab, const T* __restrict__ M,
                                                       T* __restrict__ Y, DevPlan plan = {},
                                                       const T* __restrict__ Lx = nullptr) {
    using S = GemmShape<P, T, CPLX>;
    constexpr int NC = S::NC, NE = S::NE, NCP = S::NCP, KC = S::KC;
    constexpr int JN = NCP / 16;
    constexpr bool kOneStage = KC == NE;
    const int mv = CPLX ? 2 * m : m;  // expansion rows a box
    extern __shared__ unsigned char smem_raw[];
    T* At = reinterpret_cast<T*>(smem_raw);  // [KC][NCP]: At[k][n] = A_d[n][k0 + k]
    T* Xs = At + KC * NCP;                   // [KC][64]:  Xs[k][pair]
    const int tile = blockIdx.x;
    const int d = tile_d[tile];
    const int64_t p0 = tile_begin[tile];
    const int cnt = tile_count[tile];
    const T* A = tab + (int64_t)d * NE * NE;
    // staging by asynchronous copies (every copy of the block in flight at once; padding
    // zero-filled): the table, then each vector's source rows once the tile's sources are
    // known; 256 threads
    __shared__ int32_t srcs[kGemmPairs];
    if (threadIdx.x < kGemmPairs) srcs[threadIdx.x] = threadIdx.x < cnt ? pair_src[p0 + threadIdx.x] : 0;
    auto stage_table = [&](int k0, int kc) {
        for (int t = threadIdx.x; t < kc * NCP; t += 256) {
            const int k = t / NCP, n = t % NCP;
            gemm_cp_async<T>(At + t, A + (int64_t)(k0 + k) * NE + (n < NE ? n : 0), n < NE);
        }
    };
    if (kOneStage) stage_table(0, NE);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    for (int v = blockIdx.y; v < m; v += gridDim.y) {
        const int vrow = CPLX ? 2 * v : v;
        T acc[4][JN];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < JN; ++j) acc[i][j] = T(0);
        for (int k0 = 0; k0 < NE; k0 += KC) {
            const int kc = NE - k0 < KC ? NE - k0 : KC;
            __syncthreads();  // srcs written; the previous chunk's or vector's staging read
            if (!kOneStage) stage_table(k0, kc);
            for (int t = threadIdx.x; t < kc * kGemmPairs; t += 256) {
                const int pr = t / kc, kk = k0 + t % kc;
                const int plane = CPLX ? kk / NC : 0, slot_ = CPLX ? kk % NC : kk;
                gemm_cp_async<T>(Xs + (t % kc) * kGemmPairs + pr,
                                 M + ((int64_t)srcs[pr] * mv + vrow + plane) * ms_of(P) + slot_, pr < cnt);
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_all;" ::: "memory");
            __syncthreads();
            if constexpr (sizeof(T) == 4) {
                // f32: two pairs' sums of one slot in one packed fused multiply-add (the
                // same fma a sum as the scalar loop below)
                float2 acc2[2][JN];
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < JN; ++j) acc2[i][j] = make_float2(acc[2 * i][j], acc[2 * i + 1][j]);
#pragma unroll 3
                for (int k = 0; k < kc; ++k) {
                    const float4 xv = *reinterpret_cast<const float4*>(Xs + k * kGemmPairs + ty * 4);
                    float av[JN];
#pragma unroll
                    for (int j = 0; j < JN; ++j) av[j] = At[k * NCP + tx + 16 * j];
#pragma unroll
                    for (int j = 0; j < JN; ++j) {
                        acc2[0][j] = __ffma2_rn(make_float2(av[j], av[j]), make_float2(xv.x, xv.y), acc2[0][j]);
                        acc2[1][j] = __ffma2_rn(make_float2(av[j], av[j]), make_float2(xv.z, xv.w), acc2[1][j]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < JN; ++j) {
                        acc[2 * i][j] = acc2[i][j].x;
                        acc[2 * i + 1][j] = acc2[i][j].y;
                    }
            } else {
#pragma unroll 3
                for (int k = 0; k < kc; ++k) {
                    T xv[4], av[JN];
#pragma unroll
                    for (int i = 0; i < 4; ++i) xv[i] = Xs[k * kGemmPairs + ty * 4 + i];
#pragma unroll
                    for (int j = 0; j < JN; ++j) av[j] = At[k * NCP + tx + 16 * j];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < JN; ++j) acc[i][j] += av[j] * xv[i];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int pr = ty * 4 + i;
            if (pr >= cnt) continue;
            const int64_t e = pair_e ? pair_e[p0 + pr] : p0 + pr;
            const bool x = ADD && x_of(plan, e, Lx);
            auto place = [&](int n) {
                const int plane = CPLX ? n / NC : 0, slot_ = CPLX ? n % NC : n;
                return (e * mv + vrow + plane) * ys_of(P) + slot_;
            };
            if (ADD)  // a row's locals (and X sums) read together, then added
#pragma unroll
                for (int j = 0; j < JN; ++j)
                    if (tx + 16 * j < NE) acc[i][j] += __ldcg(Y + place(tx + 16 * j));
            if (x)
#pragma unroll
                for (int j = 0; j < JN; ++j)
                    if (tx + 16 * j < NE) acc[i][j] += Lx[place(tx + 16 * j)];
#pragma unroll
            for (int j = 0; j < JN; ++j)
                if (tx + 16 * j < NE) {
                    if (ADD)
                        Y[place(tx + 16 * j)] = acc[i][j];
                    else  // read once by the reduce: stream past L2
                        __stcs(Y + place(tx + 16 * j), acc[i][j]);
                }
        }
    }
}

// ---------------------------------------------------------------------------------
// L2P + M2P of the potentials for several charge vectors (f32, m > 1): the harmonics of a
// target are formed once per W entry (and once for L2P) and dotted with VB vectors'
// expansions, which are consecutive rows of ms_of(P) floats, the harmonic rows on the packed
// f32x2 pipe and each order mu > 0 one packed fused multiply-add (real and imaginary products
// summed apart).  (Rows read 16 bytes at a time, a group of degrees in registers, were slower:
// 2.12 against 1.72 ms for 700,000 points with 16 vectors at p = 6, with 168 registers a thread.)
template <int P, int VB>
__device__ __forceinline__ void l2p_eval_mv(const float* L, int nb, float x, float y, float z, float (&f)[VB]) {
    constexpr int MS = ms_of(P);
    RegularRows2<P> h;  // the rows on the packed pipe (leaf_far_x2.cuh)
    h.init(x, y, z);
    float2 f1[VB];  // the orders mu > 0, real and imaginary products apart, weighted 2 at the end
#pragma unroll
    for (int b = 0; b < VB; ++b) {
        f[b] = 0.0f;
        f1[b] = make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int k = 0; k <= P; ++k) {
        h.step(k);
#pragma unroll
        for (int mu = 0; mu <= k; ++mu) {
#pragma unroll
            for (int b = 0; b < VB; ++b)
                if (b < nb) {
                    const Cx<float> c = coef_at(L + b * MS, k, mu);
                    if (mu == 0)
                        f[b] = fmaf(c.re, h.c[0].x, f[b]);
                    else
                        f1[b] = __ffma2_rn(make_float2(c.re, c.im), h.c[mu], f1[b]);
                }
        }
    }
#pragma unroll
    for (int b = 0; b < VB; ++b) f[b] += 2.0f * (f1[b].x - f1[b].y);
}

template <int P, int VB>
__device__ __forceinline__ void m2p_eval_mv(const float* M, int nb, float x, float y, float z, float (&f)[VB]) {
    constexpr int MS = ms_of(P);
    IrregularRows2<P> h;
    const float r2 = x * x + y * y + z * z;
    h.init(x, y, z, 1.0f / sqrt(r2));
    float2 f1[VB];
#pragma unroll
    for (int b = 0; b < VB; ++b) {
        f[b] = 0.0f;
        f1[b] = make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int k = 0; k <= P; ++k) {
        h.step(k);
#pragma unroll
        for (int mu = 0; mu <= k; ++mu) {
#pragma unroll
            for (int b = 0; b < VB; ++b)
                if (b < nb) {
                    const Cx<float> c = coef_at(M + b * MS, k, mu);
                    if (mu == 0)
                        f[b] = fmaf(c.re, h.c[0].x, f[b]);
                    else
                        f1[b] = __ffma2_rn(make_float2(c.re, c.im), h.c[mu], f1[b]);
                }
        }
    }
#pragma unroll
    for (int b = 0; b < VB; ++b) f[b] += 2.0f * (f1[b].x - f1[b].y);
}

// ---------------------------------------------------------------------------------
// What the near-field kernels share (the f64 one is near_f64.cuh, the mixed one p2p_x2.cuh,
// its near-singular pairs found by close_pairs_kernel below): a source point mapped to the
// target leaf's frame, y = fma(r, u_s, c) (CONVENTIONS 3.13 "Device kernels", rule 1), the
// pair's d = u_t - y and its r2 by explicit fma (rules 2-3), and the work items.
// ---------------------------------------------------------------------------------
constexpr int kP2pWarps = 4;
constexpr int kP2pStage = 64;

template <typename T>
__device__ __forceinline__ T map_coord(T r, T u, T c);
template <>
__device__ __forceinline__ float map_coord<float>(float r, float u, float c) { return __fmaf_rn(r, u, c); }
template <>
__device__ __forceinline__ double map_coord<double>(double r, double u, double c) { return __fma_rn(r, u, c); }

template <typename T>
__device__ __forceinline__ T pair_r2(T dx, T dy, T dz);
template <>
__device__ __forceinline__ float pair_r2<float>(float dx, float dy, float dz) {
    return __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
}
template <>
__device__ __forceinline__ double pair_r2<double>(double dx, double dy, double dz) {
    return __fma_rn(dx, dx, __fma_rn(dy, dy, __dmul_rn(dz, dz)));
}
template <typename T>
__device__ __forceinline__ T sub_rn(T a, T b);
template <>
__device__ __forceinline__ float sub_rn<float>(float a, float b) { return __fsub_rn(a, b); }
template <>
__device__ __forceinline__ double sub_rn<double>(double a, double b) { return __dsub_rn(a, b); }

struct P2pItems {
    const int32_t* leaf;  // work item -> target leaf
    const int64_t* t0;    // work item -> first target (leaf order)
    int64_t count;
    // work item -> its targets (1 to 32) | its lane slots << 8 (a power of two >= the
    // targets, 0: the targets); null: up to 32 targets, to the leaf's end, in as many slots
    const int32_t* n = nullptr;
};

// The targets ni of a work item and its slots ns: the lanes are ns targets x K = 32 / ns
// pair-step splits (lane = kk ns + ti), so an item padded to ns > ni slots splits its
// pairs as an item of ns targets would, and lanes with ti >= ni hold no target.
__device__ __forceinline__ void item_shape(const P2pItems& items, int64_t item, int64_t t1, int& ni, int& ns) {
    if (items.n) {
        const int v = items.n[item];
        ni = v & 255;
        ns = (v >> 8) ? (v >> 8) : ni;
        return;
    }
    const int64_t r = t1 - items.t0[item];
    ni = ns = (int)(r < 32 ? r : 32);
}

// L2P (own local) then M2P (W list, by box index) for every target of a leaf, over the P2P
// work items: a warp per item (up to 32 targets of one leaf, lane = target), any number of
// warps a block; a block per leaf held its whole block's registers while a leaf of few targets
// kept one warp busy.  Results (phi_hat, g_hat in the leaf's units) go to the f64 far-field
// partials.  mode: bit 0 L2P, bit 1 M2P, bit 2 add into far_phi / far_g (else overwrite them):
// the evaluation runs mode 3; the level calls run 5 (L2P) then 6 (M2P) on stores that start
// at zero, which gives the same floats.  leaf_far_mv_items_kernel forms
// each target's harmonics once for up to VB vectors (l2p_eval_mv / m2p_eval_mv).
// The gradient form is held to 96 registers up to p = 8 (21 warps an SM, no spills) and to
// 168 above (12 warps an SM; no spills to p = 12).
// With gradients (the mixed form's only use of this kernel) the terms run on the packed
// f32x2 pipe, coefficient by coefficient (l2p_x2 / m2p_x2, leaf_far_x2.cuh).
template <int P, bool GRAD>
__global__ void __launch_bounds__(128, P <= 8 ? 5 : 3) leaf_far_items_kernel(DevPlan plan, P2pItems items, int mode, int m,
                                                             const float4* __restrict__ tpos,
                                                             const float* __restrict__ M, const float* __restrict__ Lc,
                                                             double* __restrict__ far_phi, double* __restrict__ far_g) {
    static_assert(GRAD, "potentials: leaf_far_mv_items_kernel");
    const int64_t item = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= items.count) return;
    const int leaf = items.leaf[item];
    const int64_t t = items.t0[item] + (threadIdx.x & 31);
    if (t >= plan.tgt_start[leaf + 1]) return;
    const int box = plan.leaf_box[leaf];
    const int64_t w0 = plan.w_row[leaf], w1 = (mode & 2) ? plan.w_row[leaf + 1] : plan.w_row[leaf];
    const int64_t nt = plan.ntgt;
    const float4 p4 = tpos[t];
    for (int v = 0; v < m; ++v) {
        // an opaque copy of the position each vector: the harmonics are formed per
        // evaluation in registers, never hoisted out of this loop as invariants (which held
        // every row of them live across it and spilled)
        float ux = p4.x, uy = p4.y, uz = p4.z;
        asm volatile("" : "+f"(ux), "+f"(uy), "+f"(uz));
        double fphi = 0.0, fg[3] = {0.0, 0.0, 0.0};
        if (mode & 4) {
            fphi = far_phi[(int64_t)v * nt + t];
            for (int k = 0; k < 3; ++k) fg[k] = far_g[((int64_t)v * nt + t) * 3 + k];
        }
        if (mode & 1) {
            float ph, gx, gy, gz;
            l2p_x2<P, float>(Lc + ((int64_t)box * m + v) * ms_of(P), ux, uy, uz, ph, gx, gy, gz);
            fphi = (mode & 4) ? fphi + (double)ph : (double)ph;
            fg[0] = (mode & 4) ? fg[0] + (double)gx : (double)gx;
            fg[1] = (mode & 4) ? fg[1] + (double)gy : (double)gy;
            fg[2] = (mode & 4) ? fg[2] + (double)gz : (double)gz;
        }
        for (int64_t e = w0; e < w1; ++e) {
            const int s = plan.w_col[e];
            float c[3], r;
            rel_frame<float>(plan, s, box, c, r);
            const float rinv = 1.0f / r;
            float ph, gx, gy, gz;
            m2p_x2<P, float>(M + ((int64_t)s * m + v) * ms_of(P), (ux - c[0]) * rinv, (uy - c[1]) * rinv,
                      (uz - c[2]) * rinv, ph, gx, gy, gz);
            fphi += (double)(ph * rinv);
            const float r2inv = rinv * rinv;
            fg[0] += (double)(gx * r2inv);
            fg[1] += (double)(gy * r2inv);
            fg[2] += (double)(gz * r2inv);
        }
        far_phi[(int64_t)v * nt + t] = fphi;
        double* g = far_g + ((int64_t)v * nt + t) * 3;
        g[0] = fg[0];
        g[1] = fg[1];
        g[2] = fg[2];
    }
}

template <int P, int VB>
__global__ void __launch_bounds__(128) leaf_far_mv_items_kernel(DevPlan plan, P2pItems items, int mode, int m,
                                                                const float4* __restrict__ tpos,
                                                                const float* __restrict__ M,
                                                                const float* __restrict__ Lc,
                                                                double* __restrict__ far_phi) {
    constexpr int MS = ms_of(P);
    const int64_t item = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= items.count) return;
    const int leaf = items.leaf[item];
    const int64_t t = items.t0[item] + (threadIdx.x & 31);
    if (t >= plan.tgt_start[leaf + 1]) return;
    const int box = plan.leaf_box[leaf];
    const int64_t w0 = plan.w_row[leaf], w1 = (mode & 2) ? plan.w_row[leaf + 1] : plan.w_row[leaf];
    const int64_t nt = plan.ntgt;
    const float4 p4 = tpos[t];
    const float ux = p4.x, uy = p4.y, uz = p4.z;
    for (int v0 = 0; v0 < m; v0 += VB) {
        const int nb = (m - v0) < VB ? (m - v0) : VB;
        double fphi[VB];
#pragma unroll
        for (int b = 0; b < VB; ++b) fphi[b] = (b < nb && (mode & 4)) ? far_phi[(int64_t)(v0 + b) * nt + t] : 0.0;
        if (mode & 1) {
            float ph[VB];
            l2p_eval_mv<P, VB>(Lc + ((int64_t)box * m + v0) * MS, nb, ux, uy, uz, ph);
#pragma unroll
            for (int b = 0; b < VB; ++b) fphi[b] = (mode & 4) ? fphi[b] + (double)ph[b] : (double)ph[b];
        }
        for (int64_t e = w0; e < w1; ++e) {
            const int s = plan.w_col[e];
            float c[3], r;
            rel_frame<float>(plan, s, box, c, r);
            const float rinv = 1.0f / r;
            float ph[VB];
            m2p_eval_mv<P, VB>(M + ((int64_t)s * m + v0) * MS, nb, (ux - c[0]) * rinv, (uy - c[1]) * rinv,
                               (uz - c[2]) * rinv, ph);
#pragma unroll
            for (int b = 0; b < VB; ++b) fphi[b] += (double)(ph[b] * rinv);
        }
#pragma unroll
        for (int b = 0; b < VB; ++b)
            if (b < nb) far_phi[(int64_t)(v0 + b) * nt + t] = fphi[b];
    }
}

// The f64 form: a warp per item, its lanes over the item's (target, vector) pairs, target
// fastest, so that a leaf of five targets and four vectors keeps 20 lanes busy (a thread a
// target with the vectors in turn, the expansions staged in shared memory behind two block
// barriers each, kept 5).  Coefficients are read straight from global memory, the same value
// for every lane of one vector.  Each evaluation's sums do not depend on the other lanes.
// Bound by the coefficients' loads and the FP64 pipe.  Measured: 1e6 targets at p = 8 0.25 -> 0.10
// ms; 41,017 targets x 4 vectors at p = 10: see for_rows.
template <int P, bool GRAD>
__global__ void __launch_bounds__(128) leaf_far_f64_kernel(DevPlan plan, P2pItems items, int mode, int m,
                                                          const double4* __restrict__ tpos,
                                                          const double* __restrict__ M, const double* __restrict__ Lc,
                                                          double* __restrict__ far_phi, double* __restrict__ far_g) {
    const int64_t item = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= items.count) return;
    const int leaf = items.leaf[item];
    const int64_t t0 = items.t0[item], t1 = plan.tgt_start[leaf + 1];
    const int ni = t1 - t0 < 32 ? (int)(t1 - t0) : 32;
    const int box = plan.leaf_box[leaf];
    const int64_t w0 = plan.w_row[leaf], w1 = (mode & 2) ? plan.w_row[leaf + 1] : plan.w_row[leaf];
    const int64_t nt = plan.ntgt;
    for (int u = threadIdx.x & 31; u < ni * m; u += 32) {
        const int v = u / ni;
        const int64_t t = t0 + u % ni, at = (int64_t)v * nt + t;
        const double4 p4 = tpos[t];
        double fphi = 0.0, fg[3] = {0.0, 0.0, 0.0};
        if (mode & 4) {
            fphi = far_phi[at];
            if (GRAD)
                for (int k = 0; k < 3; ++k) fg[k] = far_g[at * 3 + k];
        }
        if (mode & 1) {
            const double* L = Lc + ((int64_t)box * m + v) * ms_of(P);
            double ph, gx = 0.0, gy = 0.0, gz = 0.0;
            if constexpr (GRAD) {
                l2p_x2<P, double>(L, p4.x, p4.y, p4.z, ph, gx, gy, gz);
            } else {
                RegularRows2<P, double> h;
                h.init(p4.x, p4.y, p4.z);
                ph = phi_eval<P>(h, L);
            }
            fphi += ph;
            fg[0] += gx;
            fg[1] += gy;
            fg[2] += gz;
        }
        for (int64_t e = w0; e < w1; ++e) {
            const int s = plan.w_col[e];
            double c[3], r;
            rel_frame<double>(plan, s, box, c, r);
            const double rinv = 1.0 / r;
            const double x = (p4.x - c[0]) * rinv, y = (p4.y - c[1]) * rinv, z = (p4.z - c[2]) * rinv;
            const double* Mb = M + ((int64_t)s * m + v) * ms_of(P);
            double ph, gx = 0.0, gy = 0.0, gz = 0.0;
            if constexpr (GRAD) {
                m2p_x2<P, double>(Mb, x, y, z, ph, gx, gy, gz);
            } else {
                IrregularRows2<P, double> h;
                h.init(x, y, z, 1.0 / sqrt(x * x + y * y + z * z));
                ph = phi_eval<P>(h, Mb);
            }
            fphi += ph * rinv;
            const double r2inv = rinv * rinv;
            fg[0] += gx * r2inv;
            fg[1] += gy * r2inv;
            fg[2] += gz * r2inv;
        }
        far_phi[at] = fphi;
        if (GRAD)
            for (int k = 0; k < 3; ++k) far_g[at * 3 + k] = fg[k];
    }
}

struct ClosePairs {  // near-singular pairs of the mixed form, CSR by target (leaf order)
    const int64_t* row;
    const int64_t* src;   // source point (leaf order)
    const int32_t* leaf;  // its source leaf
    const double4* spos;  // f64 leaf-scaled coordinates
    const double4* tpos;
    const double* q;      // f64 charges in leaf order [vector][point]
    const double4* y;     // the source point in the target leaf's frame (f64), per pair
    // mixed Laplace P2P: per target the f64 sum over its pairs of q times the pair's
    // weight (close_sum_kernel), [vector][target], 4 doubles (phi, grad) or 1 (phi)
    const double* acc;
};

// Build time (mixed form): each near-singular pair's source point mapped into its target
// leaf's frame in f64, y = fma(r, u, c) with the exact relative frame (the identity for the
// leaf itself), as the evaluation would form it.  Block per leaf.
static __global__ void close_map_kernel(DevPlan plan, ClosePairs close, double4* __restrict__ y) {
    const int64_t leaf = blockIdx.x;
    const int box = plan.leaf_box[leaf];
    for (int64_t t = plan.tgt_start[leaf] + threadIdx.x; t < plan.tgt_start[leaf + 1]; t += blockDim.x)
        for (int64_t c2 = close.row[t]; c2 < close.row[t + 1]; ++c2) {
            const int sl = close.leaf[c2];
            const double4 ps = close.spos[close.src[c2]];
            const double sw = (double)close.src[c2];  // w: the source's index (exact below 2^53)
            if (sl == leaf) {
                y[c2] = make_double4(ps.x, ps.y, ps.z, sw);
            } else {
                double cc[3], rr;
                rel_frame<double>(plan, plan.leaf_box[sl], box, cc, rr);
                y[c2] = make_double4(__fma_rn(rr, ps.x, cc[0]), __fma_rn(rr, ps.y, cc[1]), __fma_rn(rr, ps.z, cc[2]), sw);
            }
        }
}

// Output pass (fmm-kernels/src/movement.rs:411 gather_output with the scaling of
// fmm-exec/src/fmm.rs:4750-4778): phi = phi_hat / (4 pi r_t) and
// g = g_hat / ((4 pi r_t) r_t), leaf order -> caller order, phi_hat = far + near when the
// near field was summed apart (near_phi non-null), else the store as it is (level calls).
// Block per leaf; the same expressions as the P2P kernels' fused output, so all of them
// give the same floats.
static __global__ void output_kernel(DevPlan plan, int m, const double* __restrict__ far_phi,
                              const double* __restrict__ far_g, const double* __restrict__ near_phi,
                              const double* __restrict__ near_g, double* __restrict__ out_phi,
                              double* __restrict__ out_g) {
    const int64_t leaf = blockIdx.x;
    const int box = plan.leaf_box[leaf];
    const double rt = (plan.box_side ? plan.box_side[box] : plan.side) * pow2d(-(plan.level[box] + 1));
    const double phi_scale = 4.0 * 3.141592653589793 * rt;
    const double g_scale = phi_scale * rt;
    const int64_t nt = plan.ntgt;
    for (int v = 0; v < m; ++v)
        for (int64_t t = plan.tgt_start[leaf] + threadIdx.x; t < plan.tgt_start[leaf + 1]; t += blockDim.x) {
            const int64_t i = plan.tgt_perm[t];
            const double ph = near_phi ? far_phi[(int64_t)v * nt + t] + near_phi[(int64_t)v * nt + t]
                                       : far_phi[(int64_t)v * nt + t];
            out_phi[(int64_t)v * nt + i] = ph / phi_scale;
            if (out_g) {
                const double* fg = far_g + ((int64_t)v * nt + t) * 3;
                double* o = out_g + ((int64_t)v * nt + i) * 3;
                if (near_phi) {
                    const double* ng = near_g + ((int64_t)v * nt + t) * 3;
                    o[0] = (fg[0] + ng[0]) / g_scale;
                    o[1] = (fg[1] + ng[1]) / g_scale;
                    o[2] = (fg[2] + ng[2]) / g_scale;
                } else {
                    o[0] = fg[0] / g_scale;
                    o[1] = fg[1] / g_scale;
                    o[2] = fg[2] / g_scale;
                }
            }
        }
}

// Build time (mixed form): every near pair whose f32 r2, formed exactly as the P2P kernel
// forms it, is below theta2.  Appends (target, source point, source leaf); *count may
// exceed cap, in which case the caller enlarges the buffer and runs it again.
template <typename T>
__global__ void __launch_bounds__(128) close_pairs_kernel(DevPlan plan, P2pItems items, T theta2,
                                                          const typename Vec4<T>::type* __restrict__ spos,
                                                          const typename Vec4<T>::type* __restrict__ tpos,
                                                          unsigned long long* count, int64_t cap,
                                                          int64_t* __restrict__ out_t, int64_t* __restrict__ out_s,
                                                          int32_t* __restrict__ out_leaf) {
    using T4 = typename Vec4<T>::type;
    __shared__ T4 stage[kP2pWarps][kP2pStage];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)blockIdx.x * kP2pWarps + warp;
    if (item >= items.count) return;
    const int leaf = items.leaf[item];
    const int box = plan.leaf_box[leaf];
    const int64_t t1 = plan.tgt_start[leaf + 1];
    const int64_t t = items.t0[item] + lane;
    const bool valid = t < t1;
    T tx = T(0), ty = T(0), tz = T(0);
    if (valid) {
        T4 p4 = tpos[t];
        tx = p4.x;
        ty = p4.y;
        tz = p4.z;
    }
    for (int64_t e = plan.near_row[leaf]; e < plan.near_row[leaf + 1]; ++e) {
        const int sl = plan.near_col[e];
        T c[3] = {T(0), T(0), T(0)}, r = T(1);
        const bool self = sl == leaf;
        if (!self) rel_frame<T>(plan, plan.leaf_box[sl], box, c, r);
        const int64_t s0 = plan.src_start[sl], s1 = plan.src_start[sl + 1];
        for (int64_t sb = s0; sb < s1; sb += kP2pStage) {
            const int cnt = (int)((s1 - sb) < kP2pStage ? (s1 - sb) : kP2pStage);
            for (int j = lane; j < cnt; j += 32) {
                T4 p4 = spos[sb + j];
                T4 y;
                y.x = self ? p4.x : map_coord<T>(r, p4.x, c[0]);
                y.y = self ? p4.y : map_coord<T>(r, p4.y, c[1]);
                y.z = self ? p4.z : map_coord<T>(r, p4.z, c[2]);
                y.w = T(0);
                stage[warp][j] = y;
            }
            __syncwarp();
            if (valid)
                for (int s = 0; s < cnt; ++s) {
                    const T4 y = stage[warp][s];
                    const T dx = sub_rn<T>(tx, y.x), dy = sub_rn<T>(ty, y.y), dz = sub_rn<T>(tz, y.z);
                    if (pair_r2<T>(dx, dy, dz) < theta2) {
                        unsigned long long k = atomicAdd(count, 1ULL);
                        if ((int64_t)k < cap) {
                            out_t[k] = t;
                            out_s[k] = sb + s;
                            out_leaf[k] = sl;
                        }
                    }
                }
            __syncwarp();
        }
    }
}

}  // namespace fmmb
