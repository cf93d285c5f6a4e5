// hb_fast.cu -- the sweep kernels of the FMA FP64 stage set
// (hb_stages_fast.cuh): the same skeletons as the bit-exact FP64 kernels
// (hb_march.cuh, hb_coop.cuh).
#include "../../include/hydro_b200.h"
#include "hb_kernels.cuh"
#include "hb_march.cuh"
#include "hb_coop.cuh"
#include "hb_stages_fast.cuh"

namespace hb {

template <int DIR>
__global__ void __launch_bounds__(kSweepThreads, kFp64MarchMinBlocks)
sweep_fast_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    sweep_body<DIR, FastStages>(a, P);
}

// The warp window along rows and along columns.
template <bool NARROW>
__global__ void __launch_bounds__(kXCellThreads, kFp64WindowThreadsPerSm / kXCellThreads)
xcell_fast_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    xcell_body<FastStages, 1, NARROW>(a, P);
}
__global__ void __launch_bounds__(kYCellThreads, kFp64WindowThreadsPerSm / kYCellThreads)
ycell_fast_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    ycell_body<FastStages, kTileColumns>(a, P);
}

template <int DIR, int G>
__global__ void __launch_bounds__(kLookThreads, kLookThreadsPerSm / kLookThreads)
steady_fast_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    steady_body<FastStages, DIR, CoopShape<DIR, G>::T, CoopShape<DIR, G>::C>(a, P);
}
template <int DIR, int G>
__global__ void __launch_bounds__(CoopShape<DIR, G>::T, kCoopThreadsPerSm / CoopShape<DIR, G>::T)
coop_fast_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    coop_list_body<FastStages, DIR, CoopShape<DIR, G>::T, CoopShape<DIR, G>::C>(a, P);
}

template <int DIR, int G>
static cudaError_t launch_coop_fast_g(const SweepArgs& a, const Phys& P, cudaStream_t s) {
    using Shape = CoopShape<DIR, G>;
    return launch_coop_pair(steady_fast_kernel<DIR, G>, coop_fast_kernel<DIR, G>,
                            typename Shape::Grid(a), Shape::T, kCoopThreadsPerSm, a, P, s);
}

cudaError_t launch_sweep_fast(int dir, int kernel, const SweepArgs& a, const Phys& P,
                              cudaStream_t s) {
    if (kernel == HB_KERNEL_WARP) {
        if (dir == 2) return launch_ycells<kTileColumns>(ycell_fast_kernel, a, P, s);
        SweepArgs x = a;
        dim3 grid;
        const bool narrow = narrow_rows(x, grid);
        if (grid.y == 0) return cudaSuccess;
        launch_sweep_kernel(narrow ? xcell_fast_kernel<true> : xcell_fast_kernel<false>, grid,
                            kXCellThreads, s, x, P, kWindowCarveout);
    } else if (kernel == HB_KERNEL_COOP) {
        return dir == 1 ? launch_coop_fast_g<1, 4>(a, P, s) : launch_coop_fast_g<2, 4>(a, P, s);
    } else if (kernel == HB_KERNEL_COOP8) {
        return dir == 1 ? launch_coop_fast_g<1, 8>(a, P, s) : launch_coop_fast_g<2, 8>(a, P, s);
    } else {
        const int nl = a.n - 4;
        const int nseg = window_span(a, (nl + a.seg - 1) / a.seg);
        if (nseg == 0) return cudaSuccess;
        const dim3 grid((a.nlines + kSweepThreads - 1) / kSweepThreads, nseg);
        if (dir == 1) launch_sweep_kernel(sweep_fast_kernel<1>, grid, kSweepThreads, s, a, P);
        else launch_sweep_kernel(sweep_fast_kernel<2>, grid, kSweepThreads, s, a, P);
    }
    return cudaGetLastError();
}

int sweep_fast_blocks_per_sm(int dir) {
    int n = 0;
    cudaError_t e = dir == 1 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                                   &n, sweep_fast_kernel<1>, kSweepThreads, 0)
                             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                                   &n, sweep_fast_kernel<2>, kSweepThreads, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

__global__ void __launch_bounds__(256)
courant_fast_kernel(const double* __restrict__ u, int nx, int ny, int nxt, long long vs, Phys P,
                    unsigned long long* cour) {
    const int slot = cour_slot();
    courant_body<FastStages>(u, nx, ny, nxt, vs, P, &cour[slot], &cour[kCourSlots + slot]);
}

cudaError_t launch_courant_fast(const double* u, int nx, int ny, int nxt, long long vs,
                                const Phys& P, unsigned long long* cour, cudaStream_t s) {
    const long long total = (long long)nx * ny;
    long long blocks = (total + 255) / 256;
    const long long cap = 8ll * device_sm_count();  // 8 resident CTAs of 256 threads per SM
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    courant_fast_kernel<<<(unsigned)blocks, 256, 0, s>>>(u, nx, ny, nxt, vs, P, cour);
    return cudaGetLastError();
}

}  // namespace hb
