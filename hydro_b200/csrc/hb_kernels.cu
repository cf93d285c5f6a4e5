// hb_kernels.cu -- the fused FP64 sweep kernels and their companions.
//
// One sweep performs one dimension-split sweep (hydro_godunov.c:70-139 for one
// idim) over every interior line: boundary fill on load, primitives, slopes,
// traces, Riemann problems, fluxes and the update of each cell, in one of three
// ways to cut lines into work (all give the same bits):
//   sweep_kernel               a thread marches along a line segment with a
//                              five-cell window in registers (hb_march.cuh)
//   xcell_kernel, ycell_kernel a warp takes 32 cells of a line, one per lane
//                              (hb_march.cuh); the default below 3 Mi cells
//   steady_kernel, coop_kernel a CTA takes a window of one row or a few columns,
//                              in two launches: look, then a list (hb_coop.cuh);
//                              the default from there on
//
// Every intermediate array of the reference (u, q, c, e, dq, qxm, qxp, qleft,
// qright, qgdnv, flux, and the riemann scratch) lives in registers or shared
// memory, and HBM sees only the state: 4 doubles read and 4 written per cell and sweep
// (plus a 4-cell halo per segment or window).
//
// The sweep reads `in` and writes `out` (two buffers), so segments of one
// line can run in parallel without the read-before-overwrite hazard of the
// reference's in-place update; the host alternates the buffers so the state
// ends in the resident array after both sweeps.
#include "hb_kernels.cuh"
#include "hb_march.cuh"
#include "hb_coop.cuh"
#include "hb_batch_body.cuh"

namespace hb {

template <int DIR, bool UNIT>
__global__ void __launch_bounds__(kSweepThreads, DIR == 2 ? kFp64MarchMinBlocks : 1)
sweep_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    sweep_body<DIR, ExactStages<UNIT>>(a, P);
}

template <bool UNIT, bool NARROW>
__global__ void __launch_bounds__(kXCellThreads, kFp64WindowThreadsPerSm / kXCellThreads)
xcell_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    xcell_body<ExactStages<UNIT>, 1, NARROW>(a, P);
}

// The y sweep with one cell per lane (lanes along a column): every cell of a
// window is computed at once instead of one after another, as in a marching
// segment.  Same stage calls on the same inputs as the marcher, so the same bits.
template <bool UNIT>
__global__ void __launch_bounds__(kYCellThreads, kFp64WindowThreadsPerSm / kYCellThreads)
ycell_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    ycell_body<ExactStages<UNIT>, kTileColumns>(a, P);
}

cudaError_t launch_ycell(const SweepArgs& a, const Phys& P, cudaStream_t s) {
    return launch_ycells<kTileColumns>(P.unit_slope ? ycell_kernel<true> : ycell_kernel<false>, a, P,
                                       s);
}

// The cooperative window's two launches (hb_coop.cuh).
template <bool UNIT, int DIR, int G>
__global__ void __launch_bounds__(kLookThreads, kLookThreadsPerSm / kLookThreads)
steady_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    steady_body<ExactStages<UNIT>, DIR, CoopShape<DIR, G>::T, CoopShape<DIR, G>::C>(a, P);
}
template <bool UNIT, int DIR, int G>
__global__ void __launch_bounds__(CoopShape<DIR, G>::T, kCoopThreadsPerSm / CoopShape<DIR, G>::T)
coop_kernel(const SweepArgs a, const Phys P) {
    begin_sweep(a);
    coop_list_body<ExactStages<UNIT>, DIR, CoopShape<DIR, G>::T, CoopShape<DIR, G>::C>(a, P);
}

template <bool UNIT, int DIR, int G>
static cudaError_t launch_coop_g(const SweepArgs& a, const Phys& P, cudaStream_t s) {
    using Shape = CoopShape<DIR, G>;
    return launch_coop_pair(steady_kernel<UNIT, DIR, G>, coop_kernel<UNIT, DIR, G>,
                            typename Shape::Grid(a), Shape::T, kCoopThreadsPerSm, a, P, s);
}

template <bool UNIT>
static cudaError_t launch_coop_u(int dir, int warps, const SweepArgs& a, const Phys& P,
                                 cudaStream_t s) {
    if (warps == 8)
        return dir == 1 ? launch_coop_g<UNIT, 1, 8>(a, P, s) : launch_coop_g<UNIT, 2, 8>(a, P, s);
    return dir == 1 ? launch_coop_g<UNIT, 1, 4>(a, P, s) : launch_coop_g<UNIT, 2, 4>(a, P, s);
}

cudaError_t launch_coop(int dir, int warps, const SweepArgs& a, const Phys& P, cudaStream_t s) {
    return P.unit_slope ? launch_coop_u<true>(dir, warps, a, P, s)
                        : launch_coop_u<false>(dir, warps, a, P, s);
}

cudaError_t launch_xcell(const SweepArgs& a, const Phys& P, cudaStream_t s) {
    SweepArgs x = a;
    dim3 grid;
    const bool narrow = narrow_rows(x, grid);
    if (grid.y == 0) return cudaSuccess;
    const auto kernel = P.unit_slope ? (narrow ? xcell_kernel<true, true> : xcell_kernel<true, false>)
                                     : (narrow ? xcell_kernel<false, true> : xcell_kernel<false, false>);
    launch_sweep_kernel(kernel, grid, kXCellThreads, s, x, P, kWindowCarveout);
    return cudaGetLastError();
}

cudaError_t launch_sweep(int dir, const SweepArgs& a, const Phys& P, cudaStream_t s) {
    const int nl = a.n - 4;
    const int nseg = window_span(a, (nl + a.seg - 1) / a.seg);
    if (nseg == 0) return cudaSuccess;
    dim3 grid((a.nlines + kSweepThreads - 1) / kSweepThreads, nseg);
    if (dir == 1) {
        if (P.unit_slope) launch_sweep_kernel(sweep_kernel<1, true>, grid, kSweepThreads, s, a, P);
        else launch_sweep_kernel(sweep_kernel<1, false>, grid, kSweepThreads, s, a, P);
    } else {
        if (P.unit_slope) launch_sweep_kernel(sweep_kernel<2, true>, grid, kSweepThreads, s, a, P);
        else launch_sweep_kernel(sweep_kernel<2, false>, grid, kSweepThreads, s, a, P);
    }
    return cudaGetLastError();
}

// compute_deltat.c:54-73 as one pass over the interior: Courant speeds of
// every cell (ComputeQEforRow + equation_of_state + courantOnXY), max-reduced
// per warp and merged with atomicMax on the bit patterns (c + |u| >= 0, so
// the unsigned order of the patterns is the numeric order and max is exact).
__global__ void __launch_bounds__(256)
courant_kernel(const double* __restrict__ u, int nx, int ny, int nxt, long long vs, Phys P,
               unsigned long long* cour) {
    const int slot = cour_slot();
    courant_body<ExactStages<true>>(u, nx, ny, nxt, vs, P, &cour[slot], &cour[kCourSlots + slot]);
}

int sweep_blocks_per_sm(int dir, bool unit_slope) {
    int n = 0;
    cudaError_t e;
    if (dir == 1)
        e = unit_slope ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sweep_kernel<1, true>,
                                                                       kSweepThreads, 0)
                       : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sweep_kernel<1, false>,
                                                                       kSweepThreads, 0);
    else
        e = unit_slope ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sweep_kernel<2, true>,
                                                                       kSweepThreads, 0)
                       : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sweep_kernel<2, false>,
                                                                       kSweepThreads, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

int device_sm_count() {
    // Cached per device: the attribute does not change while the process runs.
    static int cache[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    if (cache[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
            return 1;
        cache[dev] = n;
    }
    return cache[dev];
}

cudaError_t launch_courant(const double* u, int nx, int ny, int nxt, long long vs, const Phys& P,
                           unsigned long long* cour, cudaStream_t s) {
    const long long total = (long long)nx * ny;
    long long blocks = (total + 255) / 256;
    const long long cap = 8ll * device_sm_count();  // 8 resident CTAs of 256 threads per SM
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    courant_kernel<<<(unsigned)blocks, 256, 0, s>>>(u, nx, ny, nxt, vs, P, cour);
    return cudaGetLastError();
}

// make_boundary.c:53-198 on its own (the sweeps fuse it): one thread per
// (interior line, ghost layer) of direction idim, all four variables.
__global__ void boundary_kernel(double* u, int idim, int nx, int ny, int nxt, int nyt,
                                long long vs, int bnd_lo, int bnd_hi) {
    const int nlines = (idim == 1) ? ny : nx;
    const int n = (idim == 1) ? nxt : nyt;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nlines * 4) return;
    const int l = t >> 2, gidx = t & 3;
    const int k = gidx < 2 ? gidx : n - 4 + gidx;
    const int bt = gidx < 2 ? bnd_lo : bnd_hi;
    int src;
    long long base, step;
    int mn;
    if (idim == 1) {
        src = ghost_source<1>(bt, k, n);
        base = (long long)nxt * (l + 2);
        step = 1;
        mn = 1;
    } else {
        src = ghost_source<2>(bt, k, n);
        base = l + 2;
        step = nxt;
        mn = 2;
    }
    if (src < 0) return;
    const double sn = (bt == 1) ? -1.0 : 1.0;
    for (int s = 0; s < 4; s++)
        u[base + step * k + s * vs] = u[base + step * src + s * vs] * (s == mn ? sn : 1.0);
}

cudaError_t launch_boundary(double* u, int idim, int nx, int ny, int nxt, int nyt, long long vs,
                            int bnd_lo, int bnd_hi, cudaStream_t s) {
    const int nlines = (idim == 1) ? ny : nx;
    const int threads = nlines * 4;
    boundary_kernel<<<(threads + 127) / 128, 128, 0, s>>>(u, idim, nx, ny, nxt, nyt, vs, bnd_lo,
                                                          bnd_hi);
    return cudaGetLastError();
}

// Halo strips of a domain split (make_boundary.c:48-52, mpibounds.c:165-310):
// the two interior lines next to one side, for the interior lines of the other
// direction, packed as [var][line][2] (idim 1: columns, per interior row) or
// [var][2][line] (idim 2: rows, per interior column).  Pack reads interior
// cells of `u`; unpack writes the ghost cells of the same side.  One thread per
// value; the index map is the same both ways, so unpacking a neighbour's pack
// of the opposite side puts its cells where a single grid would have them.
__global__ void halo_kernel(double* u, double* buf, int pack, int idim, int side, int nx, int ny,
                            int nxt, long long vs) {
    const int nlines = (idim == 1) ? ny : nx;
    const int total = 8 * nlines;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    int v, l, c;
    if (idim == 1) {
        c = t & 1;
        l = (t >> 1) % nlines;
        v = (t >> 1) / nlines;
    } else {
        l = t % nlines;
        c = (t / nlines) & 1;
        v = (t / nlines) >> 1;
    }
    const int nl = (idim == 1) ? nx : ny;
    // interior source line and ghost destination line along the sweep axis
    const int k_in = side == 0 ? 2 + c : nl + c;
    const int k_gh = side == 0 ? c : nl + 2 + c;
    const int k = pack ? k_in : k_gh;
    const long long at = (idim == 1) ? (long long)nxt * (l + 2) + k : (long long)nxt * k + (l + 2);
    if (pack)
        buf[t] = u[at + v * vs];
    else
        u[at + v * vs] = buf[t];
}

cudaError_t launch_halo(double* u, double* buf, int pack, int idim, int side, int nx, int ny,
                        int nxt, long long vs, cudaStream_t s) {
    const int nlines = (idim == 1) ? ny : nx;
    const int threads = 8 * nlines;
    halo_kernel<<<(threads + 255) / 256, 256, 0, s>>>(u, buf, pack, idim, side, nx, ny, nxt, vs);
    return cudaGetLastError();
}

// The maxima of the Courant slots, one pair per thread of a CTA of kCourSlots.
__device__ __forceinline__ void courant_max(unsigned long long& mx, unsigned long long& my) {
    __shared__ unsigned long long part[2][kCourSlots / 32];
    const int t = threadIdx.x;
    // c + |u| >= 0: the order of the bit patterns is the numeric order.
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xffffffffu, mx, o);
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, my, o);
        mx = mx > x ? mx : x;
        my = my > y ? my : y;
    }
    if ((t & 31) == 0) {
        part[0][t >> 5] = mx;
        part[1][t >> 5] = my;
    }
    __syncthreads();
    for (int w = 0; w < kCourSlots / 32; w++) {
        mx = mx > part[0][w] ? mx : part[0][w];
        my = my > part[1][w] ? my : part[1][w];
    }
}

// MAX(cournox, MAX(cournoy, smallc)) (compute_deltat.c:73) from the Courant
// slots, read and emptied at once by the CTA's kCourSlots threads.
__device__ __forceinline__ double take_courant_max(unsigned long long* cour, double smallc) {
    const int t = threadIdx.x;
    unsigned long long mx = cour[t], my = cour[kCourSlots + t];
    cour[t] = cour[kCourSlots + t] = 0ull;
    courant_max(mx, my);
    return omax(__longlong_as_double((long long)mx),
                omax(__longlong_as_double((long long)my), smallc));
}

// The two maxima into the host's memory, for a host that waits for them: as the
// sweep's dependent, its launch overlaps the sweep, and no copy follows it.
// With the first sweep emptying the slots, 100 steps of a 250x125 grid over the
// reference entry points, a read-back every other step: 3.50 -> 2.99 ms (a
// memset, the sweeps and a copy of every slot to pageable memory before).
__global__ void __launch_bounds__(kCourSlots)
courant_read_kernel(const unsigned long long* cour, unsigned long long* host) {
#ifdef __CUDA_ARCH__
    asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
    unsigned long long mx = cour[threadIdx.x], my = cour[kCourSlots + threadIdx.x];
    courant_max(mx, my);
    if (threadIdx.x == 0) {
        host[0] = mx;
        host[1] = my;
    }
}
cudaError_t launch_courant_read(const unsigned long long* cour, unsigned long long* host,
                                cudaStream_t s) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = 1;
    cfg.blockDim = kCourSlots;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, courant_read_kernel, cour, host);
}

// dt of an even step (main.c:349-360), halved at step 0.
__device__ __forceinline__ double even_dt(double speed, double courant_factor, double dx,
                                          int nstep) {
    double dt = courant_factor * dx / speed;
    if (nstep == 0) dt = dt / 2.0;
    return dt;
}

__device__ __forceinline__ bool clock_runs(const DevClock* c) {
    return (c->t < c->tend) && (c->nstep < c->nstepmax);
}

// main.c:407-408: nstep++, t += dt (and the dt record).
__device__ __forceinline__ void clock_advance(DevClock* c) {
    const int idx = c->nstep - c->nstep0;
    if (c->dts && idx >= 0 && idx < c->ndts) c->dts[idx] = c->dt;
    c->nstep++;
    c->t += c->dt;
}

// main.c:349-392 on the device, before a step: on even steps dt from the
// Courant maxima; stops the clock once t >= tend or nstep >= nstepmax.  The slots
// are emptied for the reduction fused into an odd step, also before one that no
// even step precedes; where the clock has stopped they keep the maxima of the
// state.  One CTA of kCourSlots threads: the slots are read at once (7 us one
// after another).
__global__ void __launch_bounds__(kCourSlots)
clock_begin_kernel(DevClock* c, unsigned long long* cour, double courant_factor, double dx,
                   double smallc) {
    const bool runs = c->active && clock_runs(c), even = (c->nstep % 2) == 0;
    double speed = 0.0;
    if (runs) speed = take_courant_max(cour, smallc);
    if (threadIdx.x != 0) return;
    if (c->active && !runs) c->active = 0;
    if (runs && even) c->dt = even_dt(speed, courant_factor, dx, c->nstep);
    c->live[0] = c->live[1] = runs;
}

// After a step.
__global__ void clock_end_kernel(DevClock* c) {
    if (c->active) clock_advance(c);
}

// The clock of an even step and the odd step after it, which takes the same
// dt, before both: whether each of them runs, and t and nstep past them.
__global__ void __launch_bounds__(kCourSlots)
clock_pair_kernel(DevClock* c, unsigned long long* cour, double courant_factor, double dx,
                  double smallc) {
    const bool runs = c->active && clock_runs(c);
    double speed = 0.0;
    if (runs) speed = take_courant_max(cour, smallc);
    if (threadIdx.x != 0) return;
    c->live[0] = runs;
    bool both = false;
    if (runs) {
        c->dt = even_dt(speed, courant_factor, dx, c->nstep);
        clock_advance(c);
        both = clock_runs(c);
        if (both) clock_advance(c);
    }
    c->live[1] = both;
    if (c->active && !both) c->active = 0;
}

cudaError_t launch_clock_begin(DevClock* c, unsigned long long* cour, double courant_factor,
                               double dx, double smallc, cudaStream_t s) {
    clock_begin_kernel<<<1, kCourSlots, 0, s>>>(c, cour, courant_factor, dx, smallc);
    return cudaGetLastError();
}

cudaError_t launch_clock_pair(DevClock* c, unsigned long long* cour, double courant_factor,
                              double dx, double smallc, cudaStream_t s) {
    clock_pair_kernel<<<1, kCourSlots, 0, s>>>(c, cour, courant_factor, dx, smallc);
    return cudaGetLastError();
}

cudaError_t launch_clock_end(DevClock* c, cudaStream_t s) {
    clock_end_kernel<<<1, 1, 0, s>>>(c);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- batches
template <bool UNIT, int DIR, int T>
__global__ void __launch_bounds__(T, (DIR == 1 ? kBatchXThreadsPerSm : kBatchYThreadsPerSm) / T)
batch_sweep_kernel(const BatchLaunch L, const Phys P) {
    batch_sweep_body<ExactStages<UNIT>, DIR, T>(L, P);
}

template <bool UNIT, int T>
static void launch_batch_t(const BatchLaunch& L, const Phys& P, int dir, int grid,
                           cudaStream_t s) {
    if (dir == 1) batch_sweep_kernel<UNIT, 1, T><<<grid, T, 0, s>>>(L, P);
    else batch_sweep_kernel<UNIT, 2, T><<<grid, T, 0, s>>>(L, P);
}

cudaError_t launch_batch_sweep(const BatchLaunch& L, const Phys& P, int dir, int grid,
                               cudaStream_t s) {
    if (L.threads == 128) {
        if (P.unit_slope) launch_batch_t<true, 128>(L, P, dir, grid, s);
        else launch_batch_t<false, 128>(L, P, dir, grid, s);
    } else {
        if (P.unit_slope) launch_batch_t<true, 64>(L, P, dir, grid, s);
        else launch_batch_t<false, 64>(L, P, dir, grid, s);
    }
    return cudaGetLastError();
}

template <class K>
static int occupancy(K kernel, int threads) {
    int n = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

template <bool UNIT, int T>
static int batch_occ(int dir) {
    return dir == 1 ? occupancy(batch_sweep_kernel<UNIT, 1, T>, T)
                    : occupancy(batch_sweep_kernel<UNIT, 2, T>, T);
}

int batch_sweep_blocks_per_sm_exact(bool unit_slope, int dir, int threads) {
    if (threads == 128) return unit_slope ? batch_occ<true, 128>(dir) : batch_occ<false, 128>(dir);
    return unit_slope ? batch_occ<true, 64>(dir) : batch_occ<false, 64>(dir);
}

// main.c:349-392 per instance (see clock_begin_kernel).
__global__ void batch_clock_begin_kernel(BatchInst* inst, int nslots, double courant_factor,
                                         double smallc, long long* gstep,
                                         unsigned int* counters) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < kBatchCounters) counters[s] = 0u;  // the step's claims
    if (s >= nslots) return;
    BatchInst& I = inst[s];
    if (!I.active) return;
    if (!((I.t < I.tend) && (I.nstep < I.nstepmax))) {
        I.active = 0;
        I.stop_step = *gstep;
        return;
    }
    if ((I.nstep % 2) == 0) {
        unsigned long long mx = 0ull, my = 0ull;
        for (int k = 0; k < kBatchCourSlots; k++) {
            mx = I.cour[k] > mx ? I.cour[k] : mx;
            my = I.cour[kBatchCourSlots + k] > my ? I.cour[kBatchCourSlots + k] : my;
            I.cour[k] = 0ull;
            I.cour[kBatchCourSlots + k] = 0ull;
        }
        const double cx = __longlong_as_double((long long)mx);
        const double cy = __longlong_as_double((long long)my);
        double dt = courant_factor * I.dx / omax(cx, omax(cy, smallc));
        if (I.nstep == 0) dt = dt / 2.0;
        I.dt = dt;
    }
}

__global__ void batch_clock_end_kernel(BatchInst* inst, int nslots, long long* gstep) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) *gstep += 1;
    if (s >= nslots) return;
    BatchInst& I = inst[s];
    if (!I.active) return;
    I.nstep++;
    I.t += I.dt;
}

cudaError_t launch_batch_clock_begin(BatchInst* inst, int nslots, double courant_factor,
                                     double smallc, long long* gstep, unsigned int* counters,
                                     cudaStream_t s) {
    batch_clock_begin_kernel<<<(nslots + 127) / 128, 128, 0, s>>>(
        inst, nslots, courant_factor, smallc, gstep, counters);
    return cudaGetLastError();
}

cudaError_t launch_batch_clock_end(BatchInst* inst, int nslots, long long* gstep,
                                   cudaStream_t s) {
    batch_clock_end_kernel<<<(nslots + 127) / 128, 128, 0, s>>>(inst, nslots, gstep);
    return cudaGetLastError();
}

// Courant maxima of the listed instances (grid y: one instance per entry).
__global__ void __launch_bounds__(256)
batch_courant_kernel(BatchInst* inst, const int* slots, int nslots, Phys P) {
    batch_courant_body<ExactStages<true>>(inst, slots, nslots, P);
}

// A single-blast initial state written on the device: density rho, zero
// momenta and energy e_bg in the interior, ghost cells 0, and energy e_blast
// in the padded cell (bi, bj) -- the layout of hydro_funcs.c:15-112.
__global__ void blast_init_kernel(double* u, int nx, int ny, double rho, double ebg, int bi,
                                  int bj, double eblast) {
    const int nxt = nx + 4, nyt = ny + 4;
    const long long vs = (long long)nxt * nyt;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < vs;
         c += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(c / nxt), i = (int)(c % nxt);
        const bool in = i >= 2 && i < nx + 2 && j >= 2 && j < ny + 2;
        u[c] = in ? rho : 0.0;
        u[c + vs] = 0.0;
        u[c + 2 * vs] = 0.0;
        u[c + 3 * vs] = in ? ((i == bi && j == bj) ? eblast : ebg) : 0.0;
    }
}

cudaError_t launch_blast_init(double* u, int nx, int ny, double rho, double ebg, int bi, int bj,
                              double eblast, cudaStream_t s) {
    const long long vs = (long long)(nx + 4) * (ny + 4);
    long long blocks = (vs + 255) / 256;
    const long long cap = 16ll * device_sm_count();
    if (blocks > cap) blocks = cap;
    blast_init_kernel<<<(unsigned)blocks, 256, 0, s>>>(u, nx, ny, rho, ebg, bi, bj, eblast);
    return cudaGetLastError();
}

cudaError_t launch_batch_courant(BatchInst* inst, const int* slots, int nslots, const Phys& P,
                                 bool mixed, cudaStream_t s) {
    if (nslots <= 0) return cudaSuccess;
    if (mixed) return launch_batch_courant_mixed(inst, slots, nslots, P, s);
    batch_courant_kernel<<<dim3(16, nslots), 256, 0, s>>>(inst, slots, nslots, P);
    return cudaGetLastError();
}

}  // namespace hb
