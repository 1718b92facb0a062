// M2M and L2L of several consecutive small levels in one launch: a cluster of eight blocks,
// block o holding octant o's table in shared memory for all of them, with a cluster barrier
// between the levels.
//
// What bounds it: latency.  A level of a few hundred boxes is a few microseconds of dependent
// work (read rows, (p+1)^2 multiply-adds, write rows), and an adaptive tree has ten such
// levels each way; as launches of their own (a product, then a reduce) each paid the table's
// load, two launches and a drain: 14 us a level at p = 6.  Levels whose children fill more
// rows than kChainRows run as launches over the whole device instead (the evaluator's
// m2m_level / l2l_level), which take over where the eight blocks' own time passes a launch's.
//
// Measured: 30,011 points in 10 levels (p = 6, f32) M2M 0.146 -> 0.082 ms, V sums and L2L
// 0.193 -> 0.116 ms, with the evaluation's 49 launches down to 20; 1e6 points of a cube (p = 8,
// f64) M2M 0.156 -> 0.096 ms.
//
// The floats are those of the separate launches: a product is the same fma chain over the
// input slots (f32) or the same fragments (f64), M2M adds a parent's products in octant order,
// L2L adds (T L_parent + S) + X with S the box's V sum, already in its local, and X its P2L sum.
//
// Rows written by one block and read by another in the same launch are read past L1 (ld.cg);
// the cluster barrier releases and acquires global memory at cluster scope.
#pragma once

#include <cooperative_groups.h>

#include "gemm_f64.cuh"
#include "kernels.cuh"

namespace fmmb {

// children x vectors of a level that stay in the chain (128 rows a block)
constexpr int64_t kChainRows = 1024;
constexpr int kChainThreads = 256;

template <int P, typename T, bool CPLX>
struct ChainShape {
    static constexpr int NC = nc_of(P), PT = CPLX ? 2 : 1;
    static constexpr int NCP = (NC + 15) / 16 * 16, XR = 34;  // f32: 32 rows a pass, padded
    static constexpr int SMEM32 = PT * NC * (NCP + XR) * 4;
    static constexpr bool OK = sizeof(T) == 8 ? GemmF64<P, CPLX>::OK && GemmF64<P, CPLX>::SPLIT == 1
                                              : SMEM32 <= 224 * 1024;
    static constexpr int SMEM = sizeof(T) == 8 ? GemmF64<P, CPLX>::SMEM : SMEM32;
};

// What a chain works on: per level and octant the pairs (child box, source box) of `pair_e`,
// `pair_src` at off[9 l + o] .. off[9 l + o + 1].
struct ChainPairs {
    const int64_t* off;
    const int64_t* pair_e;
    const int32_t* pair_src;
};

// f32: octant table(s) into shared memory as rows of input slots
template <int P, bool CPLX>
__device__ __forceinline__ void chain_table_f32(const float* __restrict__ tab, float* At) {
    using S = ChainShape<P, float, CPLX>;
    constexpr int NE = S::PT * S::NC;
    for (int i = threadIdx.x; i < S::PT * S::NC * S::NCP; i += kChainThreads) {
        const int pl = i / (S::NC * S::NCP), k = i / S::NCP % S::NC, n = i % S::NCP;
        gemm_cp_async<float>(At + i, tab + (int64_t)k * NE + pl * S::NC + (n < S::NC ? n : 0), n < S::NC);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_all;" ::: "memory");
}

// f32: rows [0, nrow) of products; row(r) -> source row pointer, put(r, n, value pair rows)
template <int P, bool CPLX, class Row, class Put>
__device__ __forceinline__ void chain_products_f32(const float* At, float* Xs, int nrow, Row&& row, Put&& put) {
    using S = ChainShape<P, float, CPLX>;
    constexpr int NC = S::NC, NCP = S::NCP, XR = S::XR, JN = NCP / 16, MS = ms_of(P), NQ = MS / 4, PT = S::PT;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    for (int r0 = 0; r0 < nrow; r0 += 32) {
        const int nr = nrow - r0 < 32 ? nrow - r0 : 32;
        __syncthreads();  // the rows of the pass before (and the table) are settled
        for (int i = threadIdx.x; i < nr * PT * NQ; i += kChainThreads) {
            const int r = i / (PT * NQ), f = i % (PT * NQ), pl = f / NQ, q = f % NQ;
            const float4 x = __ldcg(reinterpret_cast<const float4*>(row(r0 + r) + pl * MS) + q);
            float* o = Xs + (pl * NC + 4 * q) * XR + r;
            o[0] = x.x;
            if (4 * q + 1 < NC) o[XR] = x.y;
            if (4 * q + 2 < NC) o[2 * XR] = x.z;
            if (4 * q + 3 < NC) o[3 * XR] = x.w;
        }
        __syncthreads();
        float2 acc[PT][JN];
#pragma unroll
        for (int c = 0; c < PT; ++c)
#pragma unroll
            for (int j = 0; j < JN; ++j) acc[c][j] = make_float2(0.f, 0.f);
        if (2 * ty < nr) {
#pragma unroll 3
            for (int k = 0; k < NC; ++k) {
                const float2 xv = *reinterpret_cast<const float2*>(Xs + k * XR + 2 * ty);
#pragma unroll
                for (int j = 0; j < JN; ++j) {
                    const float a = At[k * NCP + tx + 16 * j];
                    acc[0][j] = __ffma2_rn(make_float2(a, a), xv, acc[0][j]);
                    if (CPLX) {
                        const float b = At[(NC + k) * NCP + tx + 16 * j];
                        acc[PT - 1][j] = __ffma2_rn(make_float2(b, b), xv, acc[PT - 1][j]);
                    }
                }
            }
            if (CPLX) {
#pragma unroll 3
                for (int k = 0; k < NC; ++k) {  // the imaginary plane: -A_i and A_r
                    const float2 xv = *reinterpret_cast<const float2*>(Xs + (NC + k) * XR + 2 * ty);
#pragma unroll
                    for (int j = 0; j < JN; ++j) {
                        const float a = At[k * NCP + tx + 16 * j], b = -At[(NC + k) * NCP + tx + 16 * j];
                        acc[0][j] = __ffma2_rn(make_float2(b, b), xv, acc[0][j]);
                        acc[PT - 1][j] = __ffma2_rn(make_float2(a, a), xv, acc[PT - 1][j]);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (2 * ty + h >= nr) break;
                for (int c = 0; c < PT; ++c)
#pragma unroll
                    for (int j = 0; j < JN; ++j) {
                        const int n = tx + 16 * j;
                        if (n < NC) put(r0 + 2 * ty + h, c, n, h ? acc[c][j].y : acc[c][j].x);
                    }
            }
        }
    }
}

// f64: the same on the FP64 tensor path; put(r, plane, n, two neighbouring values)
template <int P, bool CPLX, class Row, class Put>
__device__ __forceinline__ void chain_products_f64(const double* tab, int nrow, Row&& row, Put&& put) {
    using S = GemmF64<P, CPLX>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    constexpr int MS = ms_of(P);
    const int nrg = (nrow + 15) / 16;
    const int parts = nrg >= S::WARPS ? 1 : min(S::NG, S::WARPS / max(nrg, 1));
    for (int u = warp; u < nrg * parts; u += S::WARPS) {
        const int r0 = 16 * (u / parts) + g, r1 = r0 + 8;
        const double* a0 = r0 < nrow ? row(r0) : nullptr;
        const double* a1 = r1 < nrow ? row(r1) : nullptr;
        RowFrag<P> xr, xi;
        xr.template load<true>(a0, a1, t);
        if (CPLX) xi.template load<true>(a0 ? a0 + MS : nullptr, a1 ? a1 + MS : nullptr, t);
#pragma unroll 1
        for (int j = u % parts; j < S::NG; j += parts) {
            const int n = 8 * j + 2 * t;
            double re[4] = {0, 0, 0, 0};
            const double* br = tab + (size_t)j * S::PARTS * S::GROUP;
            xr.mul(re, br, lane);
            if constexpr (CPLX) {
                const double* bi = br + S::GROUP;
                double im[4] = {0, 0, 0, 0}, ni[4] = {0, 0, 0, 0};
                xr.mul(im, bi, lane);
                xi.mul(ni, bi, lane);
                xi.mul(im, br, lane);
#pragma unroll
                for (int q = 0; q < 4; ++q) re[q] -= ni[q];
                if (n < S::NC) {
                    if (a0) put(r0, 1, n, make_double2(im[0], im[1]));
                    if (a1) put(r1, 1, n, make_double2(im[2], im[3]));
                }
            }
            if (n < S::NC) {
                if (a0) put(r0, 0, n, make_double2(re[0], re[1]));
                if (a1) put(r1, 0, n, make_double2(re[2], re[3]));
            }
        }
    }
}

// octant o's table into shared memory (f64: packed fragments, 16 bytes a copy)
template <int P, typename T, bool CPLX>
__device__ __forceinline__ void chain_table(const T* tab, int o, unsigned char* smem) {
    if constexpr (sizeof(T) == 8) {
        using S = GemmF64<P, CPLX>;
        const double* src = tab + (size_t)o * S::TABLE;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
        for (int c = threadIdx.x; c < S::TABLE / 2; c += kChainThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * c), "l"(src + 2 * c) : "memory");
        asm volatile("cp.async.commit_group;\ncp.async.wait_all;" ::: "memory");
    } else {
        constexpr int NE = (CPLX ? 2 : 1) * nc_of(P);
        chain_table_f32<P, CPLX>(tab + (int64_t)o * NE * NE, reinterpret_cast<float*>(smem));
    }
    __syncthreads();
}

// Upward: parents of levels l_first, l_first - 1, ..., l_last from their children.  parents
// and par_start as for m2m_reduce_kernel; tab the table set of level l at l * tab_level
// elements.  A box's rows: m (PT planes each) of ms_of(P) slots.
template <int P, typename T, bool CPLX>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(kChainThreads, 1)
    chain_up_kernel(DevPlan plan, ChainPairs cp, const int32_t* __restrict__ parents,
                    const int64_t* __restrict__ par_start, int l_first, int l_last, int m,
                    const T* __restrict__ tab, int64_t tab_level, T* Yo, T* M) {
    constexpr int NC = nc_of(P), MS = ms_of(P), YS = ys_of(P), PT = CPLX ? 2 : 1;
    extern __shared__ __align__(16) unsigned char chain_smem[];
    auto cluster = cooperative_groups::this_cluster();
    const int o = (int)cluster.block_rank();
    if (tab_level == 0) chain_table<P, T, CPLX>(tab, o, chain_smem);
    for (int l = l_first; l >= l_last; --l) {
        if (tab_level != 0) {
            __syncthreads();
            chain_table<P, T, CPLX>(tab + l * tab_level, o, chain_smem);
        }
        const int64_t e0 = cp.off[9 * l + o];
        const int nrow = (int)(cp.off[9 * l + o + 1] - e0) * m;
        auto row = [&](int r) { return M + ((int64_t)cp.pair_src[e0 + r / m] * m + r % m) * (PT * MS); };
        auto out = [&](int r) { return Yo + (cp.pair_e[e0 + r / m] * m + r % m) * (PT * YS); };
        if constexpr (sizeof(T) == 8) {
            chain_products_f64<P, CPLX>(reinterpret_cast<const double*>(chain_smem), nrow, row,
                                        [&](int r, int pl, int n, double2 v) {
                                            *reinterpret_cast<double2*>(out(r) + pl * YS + n) = v;
                                        });
        } else {
            float* At = reinterpret_cast<float*>(chain_smem);
            chain_products_f32<P, CPLX>(At, At + PT * NC * ChainShape<P, T, CPLX>::NCP, nrow, row,
                                        [&](int r, int pl, int n, float v) { out(r)[pl * YS + n] = v; });
        }
        cluster.sync();
        // the parents' sums in octant order, over the cluster's threads
        const int64_t p0 = par_start[l], np = par_start[l + 1] - p0;
        const int64_t per = (int64_t)m * PT * NC;
        for (int64_t i = o * kChainThreads + threadIdx.x; i < np * per; i += 8 * kChainThreads) {
            const int p = parents[p0 + i / per], vr = (int)(i % per) / NC, n = (int)(i % NC);
            const int c0 = plan.child_first[p];
            T y[8];
#pragma unroll
            for (int c = 0; c < 8; ++c)
                y[c] = plan.src_below[c0 + c] ? __ldcg(Yo + ((int64_t)(c0 + c) * m * PT + vr) * YS + n) : T(0);
            T s = T(0);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (plan.src_below[c0 + c]) s += y[c];
            M[((int64_t)p * m * PT + vr) * MS + n] = s;
        }
        cluster.sync();
    }
}

// Downward: the children on levels l_first, l_first + 1, ..., l_last: L = (T L_parent + L) + X,
// L holding the V sum, X (when Lx is given and the box has an X list) the P2L sum.
template <int P, typename T, bool CPLX>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(kChainThreads, 1)
    chain_down_kernel(DevPlan plan, ChainPairs cp, int l_first, int l_last, int m, const T* __restrict__ tab,
                      int64_t tab_level, const T* __restrict__ Lx, T* L) {
    constexpr int NC = nc_of(P), MS = ms_of(P), PT = CPLX ? 2 : 1;
    extern __shared__ __align__(16) unsigned char chain_smem[];
    auto cluster = cooperative_groups::this_cluster();
    const int o = (int)cluster.block_rank();
    if (tab_level == 0) chain_table<P, T, CPLX>(tab, o, chain_smem);
    for (int l = l_first; l <= l_last; ++l) {
        if (tab_level != 0) {
            __syncthreads();
            chain_table<P, T, CPLX>(tab + l * tab_level, o, chain_smem);
        }
        const int64_t e0 = cp.off[9 * l + o];
        const int nrow = (int)(cp.off[9 * l + o + 1] - e0) * m;
        auto row = [&](int r) { return L + ((int64_t)cp.pair_src[e0 + r / m] * m + r % m) * (PT * MS); };
        if constexpr (sizeof(T) == 8) {
            chain_products_f64<P, CPLX>(
                reinterpret_cast<const double*>(chain_smem), nrow, row, [&](int r, int pl, int n, double2 v) {
                    const int64_t c = cp.pair_e[e0 + r / m], at = ((c * m + r % m) * PT + pl) * MS + n;
                    add_local(L + at, Lx + at, x_of(plan, c, Lx), v);
                });
        } else {
            float* At = reinterpret_cast<float*>(chain_smem);
            chain_products_f32<P, CPLX>(At, At + PT * NC * ChainShape<P, T, CPLX>::NCP, nrow, row,
                                        [&](int r, int pl, int n, float v) {
                                            const int64_t c = cp.pair_e[e0 + r / m];
                                            const int64_t at = ((c * m + r % m) * PT + pl) * MS + n;
                                            add_local(L + at, Lx + at, x_of(plan, c, Lx), v);
                                        });
        }
        cluster.sync();
    }
}

}  // namespace fmmb
