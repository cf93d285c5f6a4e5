// hb_mixed.cu -- the mixed-precision sweep kernel (stage set in
// hb_stages_mixed.cuh, march skeleton in hb_march.cuh).  Built with fast FP32
// division / square root and no FMA contraction: the stage code writes its
// fused multiply-adds out (see the Makefile).
#include "hb_kernels.cuh"
#include "hb_march.cuh"
#include "hb_coop.cuh"
#include "hb_stages_mixed.cuh"
#include "hb_batch_body.cuh"

namespace hb {

template <int DIR>
__global__ void __launch_bounds__(kSweepThreads)
sweep_mixed_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    sweep_body<DIR, MixedStages>(a, P);
}

__global__ void __launch_bounds__(kCellThreads, kMixedCellMinBlocks)
xcell_mixed_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    xcell_body<MixedStages>(a, P);
}

// Grids too small to fill the GPU take one cell per lane in both directions:
// half the chain of a two-cell x window, and a column's cells at once instead
// of one row after another.  The default's choice only (SweepArgs::one_cell: a
// kernel that the caller names is the one that runs), and for whole sweeps: the
// parts of a split sweep are counted in the other kernels' windows.  Per sweep (us, corner blast; smooth
// flow in brackets), x two cells / one, y marching / warp window:
//   250x125  12.5 (11.0) / 9.2 (9.9)     17.7 (16.9) / 9.2 (9.8)
//   512^2    12.6 (19.2) / 12.6 (18.5)   18.2 (19.6) / 14.7 (19.0)
//   724^2    13.5 (27.2) / 17.6 (27.2)   20.0 (25.1) / 25.1 (31.1)
inline bool one_cell(const SweepArgs& a) {
    return a.one_cell && a.w_lo == 0 && a.w_hi == kWholeLine;
}
__global__ void __launch_bounds__(kCellThreads, kMixedCellMinBlocks)
xcell1_mixed_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    xcell_body<MixedStages, 1>(a, P);
}
template <int NW, class Stage>
__global__ void __launch_bounds__(kCellThreads, kMixedXPipeMinBlocks)
xpipe_mixed_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    xpipe_body<MixedStages, NW, Stage>(a, P);
}

// Waits on the bulk-copy stage's mbarriers that gave up since the last call
// (g_stage_wait_timeouts of this translation unit), cleared when `reset`;
// -1 if the count cannot be read.
int mixed_stage_wait_timeouts(bool reset) {
    unsigned v = 0;
    if (cudaMemcpyFromSymbol(&v, g_stage_wait_timeouts, sizeof v) != cudaSuccess) return -1;
    if (v && reset) {
        const unsigned z = 0;
        if (cudaMemcpyToSymbol(g_stage_wait_timeouts, &z, sizeof z) != cudaSuccess) return -1;
    }
    return (int)v;
}

// The x sweep: runs of kMixedXPipeWindows pipelined windows per warp when
// they make at least four waves of the pipelined kernel's resident warps,
// else one window per warp (small grids need the parallelism more).  `bulk`
// always takes the pipelined runs, staged by bulk copies.
cudaError_t launch_xcell_mixed(const SweepArgs& a, const Phys& P, cudaStream_t s, bool bulk) {
    const int wpc = kCellThreads / 32;
    if (!bulk && one_cell(a)) {
        const int n1 = (a.n - 2 + kCellWarpOut - 1) / kCellWarpOut;
        launch_sweep_kernel(xcell1_mixed_kernel, dim3(a.nlines, (n1 + wpc - 1) / wpc),
                            kCellThreads, s, a, P, kWindowCarveout);
        return cudaGetLastError();
    }
    const int nwin =
        window_span(a, (a.n - 2 + window_out<MixedStages>() - 1) / window_out<MixedStages>());
    if (nwin == 0) return cudaSuccess;
    constexpr int NW = kMixedXPipeWindows;
    const long long runs = (long long)a.nlines * ((nwin + NW - 1) / NW);
    const dim3 pgrid(a.nlines, ((nwin + NW - 1) / NW + wpc - 1) / wpc);
    if (bulk) {
        launch_sweep_kernel(xpipe_mixed_kernel<NW, BulkWindowStage>, pgrid, kCellThreads, s, a, P);
        return cudaGetLastError();
    }
    if (runs >= 4LL * device_sm_count() * kMixedXPipeMinBlocks * wpc) {
        launch_sweep_kernel(xpipe_mixed_kernel<NW, WindowStage>, pgrid, kCellThreads, s, a, P);
        return cudaGetLastError();
    }
    dim3 grid(a.nlines, (nwin + wpc - 1) / wpc);
    launch_sweep_kernel(xcell_mixed_kernel, grid, kCellThreads, s, a, P);
    return cudaGetLastError();
}

// The cooperative window (hb_coop.cuh) with the mixed stage set, at the warp
// window's thread count per SM (kMixedCellMinBlocks CTAs of 64 threads).
constexpr int kCoopMixedThreadsPerSm = kMixedCellMinBlocks * kCellThreads;
template <int DIR, int G>
__global__ void __launch_bounds__(kLookThreads, kLookThreadsPerSm / kLookThreads)
steady_mixed_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    steady_body<MixedStages, DIR, CoopShape<DIR, G>::T, CoopShape<DIR, G>::C>(a, P);
}
template <int DIR, int G>
__global__ void __launch_bounds__(CoopShape<DIR, G>::T,
                                  kCoopMixedThreadsPerSm / CoopShape<DIR, G>::T)
coop_mixed_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    coop_list_body<MixedStages, DIR, CoopShape<DIR, G>::T, CoopShape<DIR, G>::C>(a, P);
}

template <int DIR, int G>
static cudaError_t launch_coop_mixed_g(const SweepArgs& a, const Phys& P, cudaStream_t s) {
    using Shape = CoopShape<DIR, G>;
    return launch_coop_pair(steady_mixed_kernel<DIR, G>, coop_mixed_kernel<DIR, G>,
                            typename Shape::Grid(a), Shape::T, kCoopMixedThreadsPerSm, a, P, s);
}

cudaError_t launch_coop_mixed(int dir, int warps, const SweepArgs& a, const Phys& P,
                              cudaStream_t s) {
    if (warps == 8)
        return dir == 1 ? launch_coop_mixed_g<1, 8>(a, P, s) : launch_coop_mixed_g<2, 8>(a, P, s);
    return dir == 1 ? launch_coop_mixed_g<1, 4>(a, P, s) : launch_coop_mixed_g<2, 4>(a, P, s);
}

__global__ void __launch_bounds__(kMixedYCellThreads, kMixedCellMinBlocks * kCellThreads / kMixedYCellThreads)
ycell_mixed_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    ycell_body<MixedStages, kMixedTileColumns>(a, P);
}
cudaError_t launch_sweep_mixed(int dir, const SweepArgs& a, const Phys& P, cudaStream_t s) {
    if (dir == 2 && one_cell(a)) {
        launch_sweep_kernel(ycell_mixed_kernel, ycell_grid<kMixedTileColumns>(a), kMixedYCellThreads, s,
                            a, P, kWindowCarveout);
        return cudaGetLastError();
    }
    const int nl = a.n - 4;
    const int nseg = window_span(a, (nl + a.seg - 1) / a.seg);
    if (nseg == 0) return cudaSuccess;
    dim3 grid((a.nlines + kSweepThreads - 1) / kSweepThreads, nseg);
    if (dir == 1)
        launch_sweep_kernel(sweep_mixed_kernel<1>, grid, kSweepThreads, s, a, P);
    else
        launch_sweep_kernel(sweep_mixed_kernel<2>, grid, kSweepThreads, s, a, P);
    return cudaGetLastError();
}

int sweep_mixed_blocks_per_sm(int dir) {
    int n = 0;
    cudaError_t e = dir == 1 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                                   &n, sweep_mixed_kernel<1>, kSweepThreads, 0)
                             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                                   &n, sweep_mixed_kernel<2>, kSweepThreads, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

template <int DIR, int T>
__global__ void __launch_bounds__(T, (DIR == 1 ? kBatchXMixedThreadsPerSm
                                               : kBatchYMixedThreadsPerSm) / T)
batch_sweep_mixed_kernel(const BatchLaunch L, const Phys P) {
    batch_sweep_body<MixedStages, DIR, T>(L, P);
}

cudaError_t launch_batch_sweep_mixed(const BatchLaunch& L, const Phys& P, int dir, int grid,
                                     cudaStream_t s) {
    if (L.threads == 128) {
        if (dir == 1) batch_sweep_mixed_kernel<1, 128><<<grid, 128, 0, s>>>(L, P);
        else batch_sweep_mixed_kernel<2, 128><<<grid, 128, 0, s>>>(L, P);
    } else {
        if (dir == 1) batch_sweep_mixed_kernel<1, 64><<<grid, 64, 0, s>>>(L, P);
        else batch_sweep_mixed_kernel<2, 64><<<grid, 64, 0, s>>>(L, P);
    }
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256)
courant_mixed_kernel(const double* __restrict__ u, int nx, int ny, int nxt, long long vs, Phys P,
                     unsigned long long* cour) {
    const int slot = cour_slot();
    courant_body<MixedStages>(u, nx, ny, nxt, vs, P, &cour[slot], &cour[kCourSlots + slot]);
}

cudaError_t launch_courant_mixed(const double* u, int nx, int ny, int nxt, long long vs,
                                 const Phys& P, unsigned long long* cour, cudaStream_t s) {
    const long long total = (long long)nx * ny;
    long long blocks = (total + 255) / 256;
    const long long cap = 8ll * device_sm_count();  // 8 resident CTAs of 256 threads per SM
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    courant_mixed_kernel<<<(unsigned)blocks, 256, 0, s>>>(u, nx, ny, nxt, vs, P, cour);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256)
batch_courant_mixed_kernel(BatchInst* inst, const int* slots, int nslots, Phys P) {
    batch_courant_body<MixedStages>(inst, slots, nslots, P);
}

cudaError_t launch_batch_courant_mixed(BatchInst* inst, const int* slots, int nslots,
                                       const Phys& P, cudaStream_t s) {
    batch_courant_mixed_kernel<<<dim3(16, nslots), 256, 0, s>>>(inst, slots, nslots, P);
    return cudaGetLastError();
}

int batch_sweep_blocks_per_sm_exact(bool unit_slope, int dir, int threads);  // hb_kernels.cu

template <int T>
static int batch_mixed_occ(int dir) {
    int n = 0;
    cudaError_t e = dir == 1 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                                   &n, batch_sweep_mixed_kernel<1, T>, T, 0)
                             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                                   &n, batch_sweep_mixed_kernel<2, T>, T, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

int batch_sweep_blocks_per_sm(bool mixed, bool unit_slope, int dir, int threads) {
    if (!mixed) return batch_sweep_blocks_per_sm_exact(unit_slope, dir, threads);
    return threads == 128 ? batch_mixed_occ<128>(dir) : batch_mixed_occ<64>(dir);
}

}  // namespace hb
