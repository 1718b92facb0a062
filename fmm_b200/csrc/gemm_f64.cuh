// The f64 translation products on the FP64 tensor path (mma.sync m16n8k8 / m16n8k4, f64):
// Y[pair] = A_d X[source] for pairs grouped by their table d (M2L: 316 offsets; M2M and L2L:
// 8 octants), real or complex (the Helmholtz form).
//
// What bounds it: the FP64 pipe.  A pair costs 2 (p+1)^4 flop on (p+1)^2 doubles in and out,
// so at p = 8 a pair's 13,122 flop take 0.36 ns of the chip's 37 TFLOP/s (measured here for
// m16n8k8 and for DFMA alike) and its 1.3 KB of rows 0.2 ns of HBM.  The matrix form is
// taken because a fragment feeds 32 multiply-adds a lane: a SIMT tile of 4 x 6 sums a thread
// spends as many shared-memory wavefronts as multiply-adds.
//
// Layout.  A block keeps one table in shared memory, packed as the B fragments the
// instruction wants (per 8 output slots: K-steps of 8, then a step of 4 for the odd slot of
// an even p), and walks a contiguous range of the table-sorted tile list, so that the table
// is loaded when it changes and not per tile.  A warp takes 16 rows (a row: one pair and
// vector) and loads them from global memory straight into A fragments, 16 bytes a lane:
// lane t of a row's four holds slots 2t and 2t + 1 of each 8, which is a permutation of K
// that the packed table follows.  Nothing is staged, so the warps of a block run on their
// own between table changes and one warp's gathers hide behind the others' products.
// When a block's rows of a table are few, the 8-slot column groups are dealt to the idle
// warps (a row's sums do not depend on the split).
//
// Measured: M2L of a cube of 1e6 points at p = 8 (6.0e6 V pairs) 6.35 ms on the SIMT GEMM this
// replaces, 2.3 to 2.7 ms here (30 to 34 of 37 TFLOP/s; 11 % of the products are padding of
// 81 slots to 84 x 88); whole evaluations: that cube 10.06 -> 5.96 ms, a cube of 1e5 at p = 6
// 0.608 -> 0.364, four vectors at p = 10 on 60,013 sources 3.17 -> 2.37.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "kernels.cuh"

namespace fmmb {

template <int P, bool CPLX = false>
struct GemmF64 {
    static constexpr int NC = nc_of(P);
    static constexpr int KS8 = NC / 8;                 // K-steps of 8
    static constexpr bool TAIL = NC % 8 != 0;          // NC = (p+1)^2 is 0, 1 or 4 mod 8: a step of 4
    static constexpr int NG = (NC + 7) / 8;            // groups of 8 output slots
    static constexpr int GROUP = KS8 * 64 + (TAIL ? 32 : 0);  // doubles of one group of one table
    static constexpr int PARTS = CPLX ? 2 : 1;         // A_r, A_i
    static constexpr int TABLE = NG * PARTS * GROUP;   // doubles of a packed table
    // shared memory: the whole table where it fits, else half of the column groups (blockIdx.y)
    static constexpr int SPLIT = TABLE * 8 > 220 * 1024 ? 2 : 1;
    static constexpr int NGB = (NG + SPLIT - 1) / SPLIT;
    static constexpr int SMEM = NGB * PARTS * GROUP * 8;
    static constexpr int WARPS = 8;
    // two blocks an SM where a row's fragments (2 KS8 + 1 doubles x planes) leave room
    static constexpr int BLOCKS = (PARTS * (4 * KS8 + 2) <= 42 && SMEM <= 110 * 1024) ? 2 : 1;
    // the complex form holds both planes' fragments in registers: up to p = 8
    static constexpr bool OK = !CPLX || P <= 8;
};

__device__ __forceinline__ void dmma_k8(double (&c)[4], const double (&a)[4], double b0, double b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}
__device__ __forceinline__ void dmma_k4(double (&c)[4], double a0, double a1, double b0) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},{%4,%5},{%6},{%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

// one plane of 16 rows as A fragments: lane (g, t) holds rows g and g + 8
template <int P>
struct RowFrag {
    using S = GemmF64<P>;
    double a[S::KS8 > 0 ? S::KS8 : 1][4];
    double t0, t1;
    // x0, x1: the lane's two rows (null: a row of zeros); CG: past L1 (rows that another block
    // of the launch wrote)
    template <bool CG = false>
    __device__ __forceinline__ void load(const double* x0, const double* x1, int t) {
        auto two = [](const double* x) {
            const double2* p = reinterpret_cast<const double2*>(x);
            return CG ? __ldcg(p) : *p;
        };
        auto one = [](const double* x) { return CG ? __ldcg(x) : *x; };
#pragma unroll
        for (int k = 0; k < S::KS8; ++k) {
            double2 u = make_double2(0.0, 0.0), w = u;
            if (x0) u = two(x0 + 8 * k + 2 * t);
            if (x1) w = two(x1 + 8 * k + 2 * t);
            a[k][0] = u.x;
            a[k][1] = w.x;
            a[k][2] = u.y;
            a[k][3] = w.y;
        }
        t0 = t1 = 0.0;
        if (S::TAIL && 8 * S::KS8 + t < S::NC) {
            if (x0) t0 = one(x0 + 8 * S::KS8 + t);
            if (x1) t1 = one(x1 + 8 * S::KS8 + t);
        }
    }
    // c += rows x the packed group at b (one table's KS8 steps and tail)
    __device__ __forceinline__ void mul(double (&c)[4], const double* b, int lane) const {
        const double2* b2 = reinterpret_cast<const double2*>(b) + lane;
#pragma unroll
        for (int k = 0; k < S::KS8; ++k) {
            const double2 v = b2[32 * k];
            dmma_k8(c, a[k], v.x, v.y);
        }
        if (S::TAIL) dmma_k4(c, t0, t1, b[S::KS8 * 64 + lane]);
    }
};

// Tiles: tile_d the table, tile_begin / tile_count its pairs (consecutive tiles of one table
// whose pairs follow each other are taken as one run).  Rows of pair p, vector v (plane
// pl): source row pair_src[p] * MV + MV/m v + pl of X, product row out * MV + MV/m v + pl of
// Y with out = pair_e[p] when given, else p, MV = m (2 m complex).  Rows of X are ms_of(P)
// doubles, of Y ys_of(P).
// ADD: the L2L of a level, Y = the locals: the product is added to the child's row as
// add_local does (its X sum from Lx).
template <int P, bool CPLX, bool ADD>
__global__ void __launch_bounds__(32 * GemmF64<P, CPLX>::WARPS, GemmF64<P, CPLX>::BLOCKS)
    gemm_f64_kernel(const int32_t* __restrict__ tile_d, const int64_t* __restrict__ tile_begin,
                    const int32_t* __restrict__ tile_count, int64_t ntiles, const int64_t* __restrict__ pair_e,
                    const int32_t* __restrict__ pair_src, int m, const double* __restrict__ tab,
                    const double* __restrict__ X, double* __restrict__ Y, DevPlan plan,
                    const double* __restrict__ Lx) {
    using S = GemmF64<P, CPLX>;
    static_assert(ms_of(P) == ys_of(P), "a local's row is laid out as a product's");
    constexpr int MS = ms_of(P), YS = ys_of(P), PT = S::PARTS;
    extern __shared__ __align__(16) double smem_tab[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int64_t i1 = (int64_t)(blockIdx.x + 1) * ntiles / gridDim.x;
    int64_t i = (int64_t)blockIdx.x * ntiles / gridDim.x;
    const int g0 = S::SPLIT > 1 ? (int)blockIdx.y * S::NGB : 0;  // this block's column groups
    const int ng = S::SPLIT > 1 ? min(S::NGB, S::NG - g0) : S::NG;
    int held = -1;
    while (i < i1) {
        // the run of tiles with one table, at most 32 of them, read a tile a lane
        const int64_t ti = i + lane;
        const int dd = ti < i1 ? tile_d[ti] : -1;
        const int64_t tb = ti < i1 ? tile_begin[ti] : 0;
        const int tn = ti < i1 ? tile_count[ti] : 0;
        const int d = __shfl_sync(0xffffffffu, dd, 0);
        const int64_t p0 = __shfl_sync(0xffffffffu, tb, 0);
        const int64_t before = __shfl_up_sync(0xffffffffu, tb + tn, 1);
        const unsigned follow = __ballot_sync(0xffffffffu, lane == 0 || (dd == d && tb == before));
        const int nrun = __ffs(~follow) ? __ffs(~follow) - 1 : 32;
        const int64_t p1 = __shfl_sync(0xffffffffu, tb + tn, nrun - 1);
        i += nrun;
        if (d != held) {
            __syncthreads();  // the old table is read
            const double* src = tab + (size_t)d * S::TABLE + (size_t)g0 * PT * S::GROUP;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem_tab);
            for (int c = threadIdx.x; c < ng * PT * S::GROUP / 2; c += 32 * S::WARPS)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * c), "l"(src + 2 * c)
                             : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        const int nrow = (int)(p1 - p0) * m;
        const int nrg = (nrow + 15) / 16;
        // few rows: the column groups of a row group go to `parts` warps
        const int parts = nrg >= S::WARPS ? 1 : min(ng, S::WARPS / nrg);
        const int units = nrg * parts;
        for (int u = warp; u < units || d != held; u += S::WARPS) {
            const int rg = u / parts, part = u % parts;
            const int r0 = 16 * rg + g, r1 = r0 + 8;
            RowFrag<P> xr, xi;
            const double *a0 = nullptr, *a1 = nullptr;
            int64_t o0 = 0, o1 = 0;
            bool q0 = false, q1 = false;  // ADD: the rows' boxes take an X sum
            if (u < units) {
                auto row = [&](int r, const double*& a, int64_t& o, bool& q) {
                    if (r >= nrow) return;
                    const int pr = m == 1 ? r : r / m, v = m == 1 ? 0 : r % m;
                    const int64_t p = p0 + pr;
                    a = X + ((int64_t)pair_src[p] * m + v) * (PT * MS);
                    const int64_t b = pair_e ? pair_e[p] : p;
                    o = (b * m + v) * (PT * YS);
                    q = ADD && x_of(plan, b, Lx);
                };
                row(r0, a0, o0, q0);
                row(r1, a1, o1, q1);
                xr.load(a0, a1, t);
                if (CPLX) xi.load(a0 ? a0 + MS : nullptr, a1 ? a1 + MS : nullptr, t);
            }
            if (d != held) {  // the first gathers fly while the table lands
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
                held = d;
                if (u >= units) break;
            }
            auto store = [&](int n0, const double (&c)[4], int plane) {
                const int n = n0 + 2 * t;
                if (n >= S::NC) return;
                auto put = [&](int64_t at, bool q, double2 x) {
                    if (ADD)
                        add_local(Y + at, Lx + at, q, x);
                    else  // read once by the reduce: stream past L2
                        __stcs(reinterpret_cast<double2*>(Y + at), x);
                };
                if (a0) put(o0 + plane * YS + n, q0, make_double2(c[0], c[1]));
                if (a1) put(o1 + plane * YS + n, q1, make_double2(c[2], c[3]));
            };
            if constexpr (!CPLX) {
                int j = part;
#pragma unroll 1
                for (; j + parts < ng; j += 2 * parts) {  // two groups: two independent chains
                    double c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
                    const double* b0 = smem_tab + (size_t)j * S::GROUP;
                    const double* b1 = smem_tab + (size_t)(j + parts) * S::GROUP;
                    const double2* v0 = reinterpret_cast<const double2*>(b0) + lane;
                    const double2* v1 = reinterpret_cast<const double2*>(b1) + lane;
#pragma unroll
                    for (int k = 0; k < S::KS8; ++k) {
                        const double2 e0 = v0[32 * k], e1 = v1[32 * k];
                        dmma_k8(c0, xr.a[k], e0.x, e0.y);
                        dmma_k8(c1, xr.a[k], e1.x, e1.y);
                    }
                    if (S::TAIL) {
                        dmma_k4(c0, xr.t0, xr.t1, b0[S::KS8 * 64 + lane]);
                        dmma_k4(c1, xr.t0, xr.t1, b1[S::KS8 * 64 + lane]);
                    }
                    store(8 * (g0 + j), c0, 0);
                    store(8 * (g0 + j + parts), c1, 0);
                }
                if (j < ng) {
                    double c0[4] = {0, 0, 0, 0};
                    xr.mul(c0, smem_tab + (size_t)j * S::GROUP, lane);
                    store(8 * (g0 + j), c0, 0);
                }
            } else {
                // re = A_r x_r - A_i x_i, im = A_i x_r + A_r x_i, the x_r terms first
#pragma unroll 1
                for (int j = part; j < ng; j += parts) {
                    double re[4] = {0, 0, 0, 0}, im[4] = {0, 0, 0, 0};
                    const double* br = smem_tab + (size_t)j * 2 * S::GROUP;
                    const double* bi = br + S::GROUP;
                    xr.mul(re, br, lane);
                    xr.mul(im, bi, lane);
                    double ni[4] = {0, 0, 0, 0};
                    xi.mul(ni, bi, lane);
                    xi.mul(im, br, lane);
#pragma unroll
                    for (int q = 0; q < 4; ++q) re[q] -= ni[q];
                    store(8 * (g0 + j), re, 0);
                    store(8 * (g0 + j), im, 1);
                }
            }
        }
    }
}

// Host: packs one real (p+1)^2 x (p+1)^2 table, entry (n, k) = at(n, k), as the fragments of
// gemm_f64_kernel: per 8 output slots, per K-step lane (g, t) the entries (8 j + g, 8 s + 2 t)
// and (.., + 1), then the tail's (8 j + g, 8 KS8 + t); zeros past the order.  `part` of
// `parts` interleaved tables (A_r, A_i).
template <int P, class At>
void pack_f64_table(double* out, int part, int parts, At&& at) {
    using S = GemmF64<P>;
    auto val = [&](int n, int k) { return n < S::NC && k < S::NC ? at(n, k) : 0.0; };
    for (int j = 0; j < S::NG; ++j) {
        double* o = out + ((size_t)j * parts + part) * S::GROUP;
        for (int s = 0; s < S::KS8; ++s)
            for (int l = 0; l < 32; ++l)
                for (int h = 0; h < 2; ++h) o[(s * 32 + l) * 2 + h] = val(8 * j + l / 4, 8 * s + 2 * (l % 4) + h);
        if (S::TAIL)
            for (int l = 0; l < 32; ++l) o[S::KS8 * 64 + l] = val(8 * j + l / 4, 8 * S::KS8 + l % 4);
    }
}

}  // namespace fmmb
