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
// Measured: 30,011 points in 10 levels (p = 6, f32) M2M 0.146 -> 0.058 ms, V sums and L2L
// 0.193 -> 0.091 ms, with the evaluation's 49 launches down to 20 (0.082 and 0.116 with a
// level's indexes, rows and sums read where they are needed instead of a level or a product
// ahead); 1e6 points of a cube (p = 8, f64) M2M 0.156 -> 0.088 ms.
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
    // f32: 64 rows a pass (complex: 32), a pass's rows padded by two
    static constexpr int NCP = (NC + 15) / 16 * 16, RP = CPLX ? 1 : 2, XR = 32 * RP + 2;
    static constexpr int SMEM32 = PT * NC * (NCP + XR) * 4;
    static constexpr int SMEM = sizeof(T) == 8 ? GemmF64<P, CPLX>::SMEM : SMEM32;
    // (beside the two levels' indexes, 16 KB)
    static constexpr bool OK =
        (sizeof(T) == 4 || (GemmF64<P, CPLX>::OK && GemmF64<P, CPLX>::SPLIT == 1)) && SMEM <= 210 * 1024;
};

// What a chain works on: per level and octant the pairs (child box, source box) of `pair_e`,
// `pair_src` at off[9 l + o] .. off[9 l + o + 1].
struct ChainPairs {
    const int64_t* off;
    const int64_t* pair_e;
    const int32_t* pair_src;
};

// A level's (source box, child box) of this block's octant in shared memory, two levels' worth:
// a level's are read into registers when the level before it begins and stored when it ends, so
// its rows' addresses are at hand when the cluster barrier opens.
struct ChainIndex {
    int src[kChainRows], dst[kChainRows];
    int n;
};
struct ChainNext {
    static constexpr int N = (int)(kChainRows / kChainThreads);
    int src[N], dst[N], n;
    // e0, e1: the level's pairs of this octant
    __device__ __forceinline__ void read(const ChainPairs& cp, int64_t e0, int64_t e1) {
        n = (int)(e1 - e0);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int i = threadIdx.x + j * kChainThreads;
            if (i < n) {
                src[j] = cp.pair_src[e0 + i];
                dst[j] = (int)cp.pair_e[e0 + i];
            }
        }
    }
    __device__ __forceinline__ void store(ChainIndex& ix) const {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int i = threadIdx.x + j * kChainThreads;
            if (i < n) {
                ix.src[i] = src[j];
                ix.dst[i] = dst[j];
            }
        }
        if (threadIdx.x == 0) ix.n = n;
    }
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

// f32: rows [0, nrow) of products; row(r) -> source row pointer; with ADD old(r, plane, n) -> what
// the product is added to (local, X sum), read before the sums so that its latency hides behind
// them; put(r, plane, n, product, old)
template <int P, bool CPLX, bool ADD, class Row, class Old, class Put>
__device__ __forceinline__ void chain_products_f32(const float* At, float* Xs, int nrow, Row&& row, Old&& old, Put&& put) {
    using S = ChainShape<P, float, CPLX>;
    constexpr int NC = S::NC, NCP = S::NCP, XR = S::XR, JN = NCP / 16, MS = ms_of(P), NQ = MS / 4, PT = S::PT;
    constexpr int RP = S::RP, ROWS = 32 * RP;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    for (int r0 = 0; r0 < nrow; r0 += ROWS) {
        const int nr = nrow - r0 < ROWS ? nrow - r0 : ROWS;
        __syncthreads();  // the rows of the pass before (and the table) are settled
        for (int i0 = threadIdx.x; i0 < nr * PT * NQ; i0 += 4 * kChainThreads) {  // four loads in flight
            float4 x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = i0 + j * kChainThreads, f = i % (PT * NQ);
                if (i < nr * PT * NQ)
                    x[j] = __ldcg(reinterpret_cast<const float4*>(row(r0 + i / (PT * NQ)) + f / NQ * MS) + f % NQ);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = i0 + j * kChainThreads, f = i % (PT * NQ), q = f % NQ;
                if (i >= nr * PT * NQ) break;
                float* o = Xs + (f / NQ * NC + 4 * q) * XR + i / (PT * NQ);
                o[0] = x[j].x;
                if (4 * q + 1 < NC) o[XR] = x[j].y;
                if (4 * q + 2 < NC) o[2 * XR] = x[j].z;
                if (4 * q + 3 < NC) o[3 * XR] = x[j].w;
            }
        }
        __syncthreads();
        float2 was[ADD ? RP : 1][2][ADD ? PT : 1][ADD ? JN : 1];
        if (ADD)
#pragma unroll
            for (int p = 0; p < RP; ++p)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int c = 0; c < PT; ++c)
#pragma unroll
                        for (int j = 0; j < JN; ++j) {
                            const int r = 32 * p + 2 * ty + h, n = tx + 16 * j;
                            was[p][h][c][j] = r < nr && n < NC ? old(r0 + r, c, n) : make_float2(0.f, 0.f);
                        }
        float2 acc[PT * RP][JN];  // real: a pair of rows (2 ty, 2 ty + 1) + 32 p each; complex: planes
#pragma unroll
        for (int c = 0; c < PT * RP; ++c)
#pragma unroll
            for (int j = 0; j < JN; ++j) acc[c][j] = make_float2(0.f, 0.f);
        if (2 * ty < nr) {
#pragma unroll 3
            for (int k = 0; k < NC; ++k) {
                float2 xv[RP];
#pragma unroll
                for (int p = 0; p < RP; ++p)
                    xv[p] = *reinterpret_cast<const float2*>(Xs + k * XR + 32 * p + 2 * ty);
#pragma unroll
                for (int j = 0; j < JN; ++j) {
                    const float a = At[k * NCP + tx + 16 * j];
#pragma unroll
                    for (int p = 0; p < RP; ++p) acc[p][j] = __ffma2_rn(make_float2(a, a), xv[p], acc[p][j]);
                    if (CPLX) {
                        const float b = At[(NC + k) * NCP + tx + 16 * j];
                        acc[PT - 1][j] = __ffma2_rn(make_float2(b, b), xv[0], acc[PT - 1][j]);
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
            for (int p = 0; p < RP; ++p)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = 32 * p + 2 * ty + h;
                    if (r >= nr) continue;
#pragma unroll
                    for (int c = 0; c < PT; ++c)
#pragma unroll
                        for (int j = 0; j < JN; ++j) {
                            const int n = tx + 16 * j;
                            const float2 v = acc[CPLX ? c : p][j];
                            if (n < NC)
                                put(r0 + r, c, n, h ? v.y : v.x, ADD ? was[p][h][c][j] : make_float2(0.f, 0.f));
                        }
                }
        }
    }
}

// f64: the same on the FP64 tensor path, two neighbouring slots at a time: old(r, plane, n, l, x)
template <int P, bool CPLX, bool ADD, class Row, class Old, class Put>
__device__ __forceinline__ void chain_products_f64(const double* tab, int nrow, Row&& row, Old&& old, Put&& put) {
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
            const double2 z = make_double2(0.0, 0.0);
            double2 l[S::PARTS][2], x[S::PARTS][2];
#pragma unroll
            for (int c = 0; c < S::PARTS; ++c) {
                l[c][0] = l[c][1] = x[c][0] = x[c][1] = z;
                if (ADD && n < S::NC) {
                    if (a0) old(r0, c, n, l[c][0], x[c][0]);
                    if (a1) old(r1, c, n, l[c][1], x[c][1]);
                }
            }
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
                    if (a0) put(r0, 1, n, make_double2(im[0], im[1]), l[1][0], x[1][0]);
                    if (a1) put(r1, 1, n, make_double2(im[2], im[3]), l[1][1], x[1][1]);
                }
            }
            if (n < S::NC) {
                if (a0) put(r0, 0, n, make_double2(re[0], re[1]), l[0][0], x[0][0]);
                if (a1) put(r1, 0, n, make_double2(re[2], re[3]), l[0][1], x[0][1]);
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

// Upward: parents of levels l_first, l_first - 1, ..., l_last from their children.  par_rec the
// M2M parents by level (par_start): the parent, its first child, the bits of its children that
// hold a source; tab the table set of level l at l * tab_level
// elements.  A box's rows: m (PT planes each) of ms_of(P) slots.
template <int P, typename T, bool CPLX>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(kChainThreads, 1)
    chain_up_kernel(ChainPairs cp, const int4* __restrict__ par_rec, const int64_t* __restrict__ par_start, int l_first, int l_last, int m,
                    const T* __restrict__ tab, int64_t tab_level, T* Yo, T* M) {
    constexpr int NC = nc_of(P), MS = ms_of(P), YS = ys_of(P), PT = CPLX ? 2 : 1;
    extern __shared__ __align__(16) unsigned char chain_smem[];
    auto cluster = cooperative_groups::this_cluster();
    __shared__ ChainIndex index[2];
    const int o = (int)cluster.block_rank();
    ChainNext next;
    next.read(cp, cp.off[9 * l_first + o], cp.off[9 * l_first + o + 1]);
    next.store(index[0]);
    const int per = m * PT * NC;  // values of a parent
    const int64_t first = o * kChainThreads + threadIdx.x;
    // the next level's pairs and this level's parents: their ranges read a level ahead
    int64_t e0 = l_first > l_last ? cp.off[9 * (l_first - 1) + o] : 0;
    int64_t e1 = l_first > l_last ? cp.off[9 * (l_first - 1) + o + 1] : 0;
    int64_t p0 = par_start[l_first], p1 = par_start[l_first + 1];
    if (tab_level == 0) chain_table<P, T, CPLX>(tab, o, chain_smem);  // (ends with a block barrier)
    for (int l = l_first; l >= l_last; --l) {
        if (tab_level != 0) {
            __syncthreads();
            chain_table<P, T, CPLX>(tab + l * tab_level, o, chain_smem);
        }
        // what does not wait for this level's products is read beside them
        const int64_t np = p1 - p0, base = p0;
        int4 rec = first < np * per ? par_rec[base + first / per] : make_int4(0, 0, 0, 0);
        if (l > l_last) {
            next.read(cp, e0, e1);
            p1 = p0;
            p0 = par_start[l - 1];
            if (l - 1 > l_last) {
                e0 = cp.off[9 * (l - 2) + o];
                e1 = cp.off[9 * (l - 2) + o + 1];
            }
        }
        const ChainIndex& ix = index[(l_first - l) & 1];
        const int nrow = (int)ix.n * m;
        auto row = [&](int r) { return M + ((int64_t)ix.src[r / m] * m + r % m) * (PT * MS); };
        auto out = [&](int r) { return Yo + ((int64_t)ix.dst[r / m] * m + r % m) * (PT * YS); };
        if constexpr (sizeof(T) == 8) {
            chain_products_f64<P, CPLX, false>(
                reinterpret_cast<const double*>(chain_smem), nrow, row,
                [](int, int, int, double2&, double2&) {},
                [&](int r, int pl, int n, double2 v, double2, double2) {
                    *reinterpret_cast<double2*>(out(r) + pl * YS + n) = v;
                });
        } else {
            float* At = reinterpret_cast<float*>(chain_smem);
            chain_products_f32<P, CPLX, false>(
                At, At + PT * NC * ChainShape<P, T, CPLX>::NCP, nrow, row,
                [](int, int, int) { return make_float2(0.f, 0.f); },
                [&](int r, int pl, int n, float v, float2) { out(r)[pl * YS + n] = v; });
        }
        if (l > l_last) next.store(index[(l_first - l + 1) & 1]);
        cluster.sync();
        // the parents' sums in octant order, over the cluster's threads
        for (int64_t i = first; i < np * per; i += 8 * kChainThreads) {
            if (i != first) rec = par_rec[base + i / per];
            const int vr = (int)(i % per) / NC, n = (int)(i % per) % NC;
            T y[8];
#pragma unroll
            for (int c = 0; c < 8; ++c)
                y[c] = rec.z >> c & 1 ? __ldcg(Yo + ((int64_t)(rec.y + c) * m * PT + vr) * YS + n) : T(0);
            T s = T(0);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (rec.z >> c & 1) s += y[c];
            M[((int64_t)rec.x * m * PT + vr) * MS + n] = s;
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
    __shared__ ChainIndex index[2];
    const int o = (int)cluster.block_rank();
    ChainNext next;
    next.read(cp, cp.off[9 * l_first + o], cp.off[9 * l_first + o + 1]);
    next.store(index[0]);
    int64_t e0 = l_first < l_last ? cp.off[9 * (l_first + 1) + o] : 0;
    int64_t e1 = l_first < l_last ? cp.off[9 * (l_first + 1) + o + 1] : 0;
    if (tab_level == 0) chain_table<P, T, CPLX>(tab, o, chain_smem);  // (ends with a block barrier)
    for (int l = l_first; l <= l_last; ++l) {
        if (tab_level != 0) {
            __syncthreads();
            chain_table<P, T, CPLX>(tab + l * tab_level, o, chain_smem);
        }
        if (l < l_last) {  // the next level's pairs, read beside this level's products
            next.read(cp, e0, e1);
            if (l + 1 < l_last) {
                e0 = cp.off[9 * (l + 2) + o];
                e1 = cp.off[9 * (l + 2) + o + 1];
            }
        }
        const ChainIndex& ix = index[(l - l_first) & 1];
        const int nrow = (int)ix.n * m;
        auto row = [&](int r) { return L + ((int64_t)ix.src[r / m] * m + r % m) * (PT * MS); };
        if constexpr (sizeof(T) == 8) {
            chain_products_f64<P, CPLX, true>(
                reinterpret_cast<const double*>(chain_smem), nrow, row,
                [&](int r, int pl, int n, double2& l0, double2& x0) {
                    const int64_t c = ix.dst[r / m], at = ((c * m + r % m) * PT + pl) * MS + n;
                    l0 = __ldcg(reinterpret_cast<const double2*>(L + at));
                    if (x_of(plan, c, Lx)) x0 = *reinterpret_cast<const double2*>(Lx + at);
                },
                [&](int r, int pl, int n, double2 v, double2 l0, double2 x0) {
                    const int64_t c = ix.dst[r / m], at = ((c * m + r % m) * PT + pl) * MS + n;
                    *reinterpret_cast<double2*>(L + at) = make_double2((v.x + l0.x) + x0.x, (v.y + l0.y) + x0.y);
                });
        } else {
            float* At = reinterpret_cast<float*>(chain_smem);
            chain_products_f32<P, CPLX, true>(
                At, At + PT * NC * ChainShape<P, T, CPLX>::NCP, nrow, row,
                [&](int r, int pl, int n) {
                    const int64_t c = ix.dst[r / m], at = ((c * m + r % m) * PT + pl) * MS + n;
                    return make_float2(__ldcg(L + at), x_of(plan, c, Lx) ? Lx[at] : 0.f);
                },
                [&](int r, int pl, int n, float v, float2 was) {
                    const int64_t c = ix.dst[r / m];
                    L[((c * m + r % m) * PT + pl) * MS + n] = (v + was.x) + was.y;
                });
        }
        if (l < l_last) next.store(index[(l - l_first + 1) & 1]);
        cluster.sync();
    }
}

}  // namespace fmmb
