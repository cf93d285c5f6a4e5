// hb_kernels.cuh -- kernel argument records and launchers shared by the
// host runtime (hb_runtime.cu) and the kernels (hb_kernels.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "hb_stages.cuh"

namespace hb {

// Device-resident clock of the multi-step driver (main.c:344-408 state).
struct DevClock {
    double t, dt, tend;
    int nstep, nstepmax;
    int nstep0;   // nstep when the clock was last set (index base of dts)
    int active;   // 0 once t >= tend or nstep >= nstepmax
    int live[2];  // whether the sweeps of the even / odd step of a pair run
    double* dts;  // optional per-step dt record
    int ndts;
};

// One fused sweep over every interior line of a direction.
struct SweepArgs {
    const double* in;        // interior cells are read here
    const double* resid;     // the resident state: ghost cells are read (and sourced) here
                             // when they are not interior cells
    double* out;             // updated interior cells are written here
    double* gout;            // ghost cells of the swept direction are written here (or null)
    const DevClock* clk;     // null: use dt below; else dt and whether to run come from here
    int odd;                 // the step's parity: which of clk->live counts
    double dt;
    unsigned long long* courant;  // null or [2 * kCourSlots] fused maxima (bit patterns)
    int nx, ny, nxt, nyt;
    long long vs;            // nxt * nyt (stride between variables)
    int bnd_lo, bnd_hi;      // boundary types of the swept direction (left/right or down/up)
    int seg;                 // output cells per thread segment
    int nlines;              // interior lines (ny for the x sweep, nx for the y sweep)
    int n;                   // cells along a line including ghosts (nxt or nyt)
    // Windows (segments for the marching kernels) [w_lo, w_hi) of every line
    // are swept: the launch grid starts at window w_lo.  0 and a large w_hi
    // sweep the whole line; a domain split sweeps the windows that read no
    // ghost cell while the halos travel, and the others after.
    int w_lo, w_hi;
    int row_shift;  // x warp windows of narrow rows (narrow_rows)
    int one_cell;  // mixed: the default of a small grid (kOneCellMixedMaxCells)
    // The cooperative sweeps' list of windows (hb_coop.cuh; room for every
    // window of a sweep), and its length, a ticket and the claims made on it,
    // all 0 between sweeps.
    int2* todo;
    unsigned* todo_count;
    // null, or the [2 * kCourSlots] maxima to empty before the sweep (a
    // dependent's first CTA does; the test sits there because in the short CTAs
    // of a captured sweep it cost 2%, 1024^2 at rest).
    unsigned long long* empty;
    int dependent;  // launched as a programmatic dependent (launch_sweep_kernel)
};

// Windows of [w_lo, w_hi) n [0, total) a launch covers (its grid's y extent
// in windows; 0: nothing to launch).
inline int window_span(const SweepArgs& a, int total) {
    const int hi = a.w_hi < total ? a.w_hi : total;
    return hi > a.w_lo ? hi - a.w_lo : 0;
}
constexpr int kWholeLine = 1 << 30;  // w_hi of a launch over whole lines

constexpr int kSweepThreads = 64;

// The fused Courant maxima are accumulated with atomicMax into kCourSlots
// slots per direction ([0, kCourSlots): max(c+|u|), [kCourSlots, 2*kCourSlots):
// max(c+|v|)), the slot chosen by the CTA index, so that no single address
// takes one atomic per warp of the whole grid; readers take the max over the
// slots (max is exact, so the result does not depend on the split).
constexpr int kCourSlots = 128;

// Sweep kernels launched one by one into a stream are programmatic dependents:
// the next one's launch overlaps the tail of the one before, and each of its
// CTAs begins by waiting until all work before it is complete and visible
// (begin_sweep).  Two steps of a 250x125 grid through the allocation-free entry
// point, four 10 us sweeps: 46.9 -> 38.6 us.  Into a capture they are launched
// as ordinary nodes: a graph starts its kernels about as early by itself, and
// its step pairs were 2% slower with the wait in their many small CTAs.  State
// and clock are read by ordinary loads (the read-only path wants data that no
// kernel in flight writes).
__device__ __forceinline__ void begin_sweep(const SweepArgs& a) {
#ifdef __CUDA_ARCH__
    if (a.dependent) {
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (a.empty && blockIdx.x == 0 && blockIdx.y == 0)
            for (int i = threadIdx.x; i < 2 * kCourSlots; i += blockDim.x) a.empty[i] = 0ull;
    }
#endif
}
inline cudaError_t launch_sweep_kernel(void (*kernel)(SweepArgs, Phys), dim3 grid, int threads,
                                       cudaStream_t s, SweepArgs a, const Phys& P,
                                       int carveout = -1) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const cudaError_t e = cudaStreamIsCapturing(s, &capture);
    if (e != cudaSuccess) return e;
    a.dependent = capture == cudaStreamCaptureStatusNone;
    if (a.empty && !a.dependent) {
        const cudaError_t m =
            cudaMemsetAsync(a.empty, 0, 2 * kCourSlots * sizeof(*a.empty), s);
        if (m != cudaSuccess) return m;
    }
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (a.dependent) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (carveout >= 0) {
        attr[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        attr[n++].val.sharedMemCarveout = (unsigned)carveout;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = threads;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, a, P);
}

// Multiprocessor count of the current device (cudaDevAttrMultiProcessorCount,
// cached per device; 1 if it cannot be read).
int device_sm_count();

// Launchers (hb_kernels.cu).  Each returns the cudaError_t of the launch.
cudaError_t launch_sweep(int dir, const SweepArgs& a, const Phys& P, cudaStream_t s);
// Resident sweep CTAs per SM (cudaOccupancyMaxActiveBlocksPerMultiprocessor).
int sweep_blocks_per_sm(int dir, bool unit_slope);
// The mixed x sweep's windows (hb_march.cuh xcell_body, xpipe_body).
constexpr int kCellThreads = 64;
// The FP64 / FMA x warp windows take 8 warps a CTA (a CTA of 2 was bound by
// CTA launches at rest: 1024^2 27.7 -> 23.5 us).
constexpr int kXCellThreads = 256;
// Columns of the y form's tiles, one warp each.  FP64 / FMA: 8 (64-byte runs),
// against 4 (32 bytes): at 1024^2 energy noise 78.3 -> 75.0 us, a centred blast
// 27.3 -> 23.0, 3001 x 777 noise 160 -> 154; 250 x 125 noise 14.7 -> 15.3.  The
// mixed form runs on small grids alone, where CTAs are few: 4 (512^2 17.5 us,
// 18.7 with 8).  A batch's y items: one warp takes the 4 columns of its tile.
constexpr int kTileColumns = 8;
constexpr int kMixedTileColumns = 4;
constexpr int kBatchTileColumns = 4;
constexpr int kYCellThreads = 32 * kTileColumns;
constexpr int kMixedYCellThreads = 32 * kMixedTileColumns;
// The share of an SM's L1 (percent) both directions' warp windows ask for as
// shared memory.  A kernel that wants another split than the one before it
// waits until the SM has drained: with x (no shared memory) and y (tiles) left
// to their own defaults, four dependent sweeps of 250 x 125 took 51 us, 42 with
// one split for both (20 ... 50 % alike).
constexpr int kWindowCarveout = 25;

// Minimum resident CTAs per SM the sweep kernels are compiled for (register
// caps).  The FP64 kernels are latency-bound: more resident warps beat the
// few register spills the caps cause.  The FP64 / FMA warp windows hold 1024
// threads an SM (64 registers, 96 bytes of spills; 4 CTAs of 256): 1024^2 41
// steps of a blast 1827 us so, 1927 and 1921 with CTAs of 64 and 128.  The marching
// y sweep 16 CTAs of 64 (4096^2 1.66 -> 1.49 ms).  The mixed marching
// sweep is not capped; the mixed x sweep (two cells per lane) runs best at 12
// CTAs per SM (80 registers): 0.419 ms at 4096^2, against 0.477 ms one cell
// per lane.
constexpr int kFp64MarchMinBlocks = 16;
constexpr int kFp64WindowThreadsPerSm = 1024;
constexpr int kMixedCellMinBlocks = 12;
// The software-pipelined mixed x sweep (xpipe_body): two-cell windows per warp
// and its register cap (8 CTAs of 64 per SM: 119 registers, no spills).  At
// 4096^2: 0.258 ms with runs of 6 windows, 0.267 with 8, 0.268 with 4, 0.304
// with 2 (at 12 CTAs per SM and 80 registers, runs of 4: 0.291 ms), against
// 0.309 ms for one window per warp.
constexpr int kMixedXPipeWindows = 6;
constexpr int kMixedXPipeMinBlocks = 8;
// The FP64 cooperative windows (hb_coop.cuh): resident threads per SM their
// two launches are compiled for.  At 4096^2, x + y, with 1152 / 1024 / 896 / 768
// threads of the second launch: energy noise 2046 / 2041 / 2084 / 2089 us,
// centred blast 420 / 422 / 421 / 426 us (1152 is 1024 along y, whose CTAs have
// 256 threads).
constexpr int kCoopThreadsPerSm = 1024;
constexpr int kLookThreadsPerSm = 1024;
// Outputs per line of a cooperative window (G = 4 or 8 warps along x).
__host__ __device__ constexpr int coop_outputs(int dir, int g) {
    return dir == 1 ? 32 * g - 4 : (g == 4 ? 60 : 124);
}
// Windows of the domain's cooperative sweeps at most (the narrowest outputs).
inline long long coop_list_size(int nx, int ny) {
    const long long x = (long long)ny * ((nx + 2 + coop_outputs(1, 4) - 1) / coop_outputs(1, 4));
    const long long y4 = (nx + 2 + 3) / 4 * (long long)((ny + 2 + coop_outputs(2, 4) - 1) / coop_outputs(2, 4));
    const long long y8 = (nx + 2 + 1) / 2 * (long long)((ny + 2 + coop_outputs(2, 8) - 1) / coop_outputs(2, 8));
    return x > y4 ? (x > y8 ? x : y8) : (y4 > y8 ? y4 : y8);
}
// Grids of at most this many cells take one cell per lane in both directions by
// default in mixed precision (hb_mixed.cu).
constexpr long long kOneCellMixedMaxCells = 1ll << 18;
constexpr int kCellWarpOut = 28;   // outputs per warp of the cell-per-lane x sweep
constexpr int kCellWarpOut2 = 60;  // the same with two cells per lane
// Outputs per warp of the x sweep window of a stage set.
template <class S>
constexpr int window_out() { return S::cells_per_lane == 2 ? kCellWarpOut2 : kCellWarpOut; }
cudaError_t launch_xcell(const SweepArgs& a, const Phys& P, cudaStream_t s);
// The cooperative window (hb_coop.cuh), `warps` = 4 or 8 warps per CTA.
cudaError_t launch_coop(int dir, int warps, const SweepArgs& a, const Phys& P, cudaStream_t s);
cudaError_t launch_coop_mixed(int dir, int warps, const SweepArgs& a, const Phys& P,
                              cudaStream_t s);
cudaError_t launch_ycell(const SweepArgs& a, const Phys& P, cudaStream_t s);
// The mixed x sweep (two-cell windows); `bulk`: staged by TMA-engine bulk
// copies (HB_KERNEL_BULK) instead of per-lane cp.async.
cudaError_t launch_xcell_mixed(const SweepArgs& a, const Phys& P, cudaStream_t s,
                               bool bulk = false);
// Waits of the mixed x sweep's bulk-copy stage that gave up (hb_mixed.cu).
int mixed_stage_wait_timeouts(bool reset);
// The FMA FP64 stage set (hb_fast.cu): kernel = HB_KERNEL_* (include/hydro_b200.h).
cudaError_t launch_sweep_fast(int dir, int kernel, const SweepArgs& a, const Phys& P,
                              cudaStream_t s);
int sweep_fast_blocks_per_sm(int dir);
cudaError_t launch_courant_fast(const double* u, int nx, int ny, int nxt, long long vs,
                                const Phys& P, unsigned long long* cour, cudaStream_t s);
// The mixed-precision sweep (hb_mixed.cu).
cudaError_t launch_sweep_mixed(int dir, const SweepArgs& a, const Phys& P, cudaStream_t s);
int sweep_mixed_blocks_per_sm(int dir);
cudaError_t launch_courant(const double* u, int nx, int ny, int nxt, long long vs, const Phys& P,
                           unsigned long long* cour, cudaStream_t s);
cudaError_t launch_courant_mixed(const double* u, int nx, int ny, int nxt, long long vs,
                                 const Phys& P, unsigned long long* cour, cudaStream_t s);
cudaError_t launch_boundary(double* u, int idim, int nx, int ny, int nxt, int nyt, long long vs,
                            int bnd_lo, int bnd_hi, cudaStream_t s);
cudaError_t launch_vtk_base64(const double* var_plane, int nx, int ny, int nxt,
                              unsigned char* out, cudaStream_t s);
cudaError_t launch_halo(double* u, double* buf, int pack, int idim, int side, int nx, int ny,
                        int nxt, long long vs, cudaStream_t s);
cudaError_t launch_courant_read(const unsigned long long* cour, unsigned long long* host,
                                cudaStream_t s);
cudaError_t launch_clock_begin(DevClock* c, unsigned long long* cour, double courant_factor,
                               double dx, double smallc, cudaStream_t s);
cudaError_t launch_clock_end(DevClock* c, cudaStream_t s);
cudaError_t launch_clock_pair(DevClock* c, unsigned long long* cour, double courant_factor,
                              double dx, double smallc, cudaStream_t s);

}  // namespace hb
