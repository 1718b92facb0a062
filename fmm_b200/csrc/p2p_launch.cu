// The launches of the near-field kernels that do not depend on the expansion order (the
// streamed mixed P2P, the f64 near field), in a translation unit of their own: compiled once,
// not once per order.
#include "near_f64.cuh"
#include "p2p_x2.cuh"

namespace fmmb {

namespace {
template <int W, int KS>
void launch_wk(const P2pStArgs& a, unsigned grid, cudaStream_t s) {
    if (a.m == 1)
        p2p_st_kernel<true, W, true, KS><<<grid, 32 * W, 0, s>>>(a);
    else
        p2p_st_kernel<true, W, false, KS><<<grid, 32 * W, 0, s>>>(a);
}

template <int W>
void launch_w(const P2pStArgs& a, int ks, unsigned grid, cudaStream_t s) {
    switch (ks) {
        case 1: launch_wk<W, 1>(a, grid, s); break;
        case 2: launch_wk<W, 2>(a, grid, s); break;
        case 4: launch_wk<W, 4>(a, grid, s); break;
        case 8: launch_wk<W, 8>(a, grid, s); break;
        default: launch_wk<W, 0>(a, grid, s);
    }
}
}  // namespace

void launch_p2p_st(const P2pStArgs& a, int warps, int ks, unsigned grid, cudaStream_t s) {
    if (warps == 1)
        launch_w<1>(a, ks, grid, s);
    else if (warps == 2)
        launch_w<2>(a, ks, grid, s);
    else
        launch_w<4>(a, ks, grid, s);
}

namespace {
// Warps an item: 8, 4 or 2 while the items alone would leave most of an SM's schedulers
// without a warp (an SM wants about eight of the kernel's warps to be busy), else a warp an
// item.  The floats are the same either way.
template <class PK>
void launch_near(const NearArgs& a, cudaStream_t s) {
    const int64_t n = a.items.count;
    const size_t stage = sizeof(double) * near_stage_doubles<PK>() * kNearFlush;
    const int w = n <= 2 * a.num_sms ? 8 : n <= 4 * a.num_sms ? 4 : n <= 8 * a.num_sms ? 2 : 1;
    if (w > 1)
        near_f64_kernel<PK, true><<<(unsigned)n, 32 * w, w * stage, s>>>(a);
    else
        near_f64_kernel<PK, false>
            <<<(unsigned)((n + kNearWarps - 1) / kNearWarps), 32 * kNearWarps, kNearWarps * stage, s>>>(a);
}
template <bool GRAD>
void launch_near_vectors(const NearArgs& a, cudaStream_t s) {
    if (a.m == 1)
        launch_near<NearLaplace<GRAD, 1>>(a, s);
    else if (a.m == 2)
        launch_near<NearLaplace<GRAD, 2>>(a, s);
    else
        launch_near<NearLaplace<GRAD, 4>>(a, s);
}
}  // namespace

void launch_near_laplace_f64(const NearArgs& a, bool gradients, cudaStream_t s) {
    if (gradients)
        launch_near_vectors<true>(a, s);
    else
        launch_near_vectors<false>(a, s);
}

void launch_near_helmholtz_f64(const NearArgs& a, bool gradients, cudaStream_t s) {
    if (gradients)
        launch_near<NearHelmholtz<true>>(a, s);
    else
        launch_near<NearHelmholtz<false>>(a, s);
}

}  // namespace fmmb
