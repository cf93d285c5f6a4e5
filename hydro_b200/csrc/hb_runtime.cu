// hb_runtime.cu -- host runtime and C ABI of libhydro_b200.so.
//
// Layers:
//   hb_domain          a device-resident state (reference layout), its scratch
//                      buffer, Courant accumulators, device clock and stream;
//   reference ABI      hydro_godunov / compute_deltat / make_boundary / ... with
//                      the reference's signatures, mapping Hv->uold to a
//                      domain through a registry (device mirror of host memory);
//   hydro_b200_*       residency control, the device-resident driver loop,
//                      errors, and the domain (device pointer) API.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "../../include/hydro_b200.h"
#include "hb_kernels.cuh"

using hb::DevClock;
using hb::Phys;
using hb::SweepArgs;

static constexpr size_t kCourBytes = 2 * hb::kCourSlots * sizeof(unsigned long long);
static constexpr long long kCoopMinCells = 3ll << 20;     // see default_kernel
static constexpr long long kCoopMinCellsFma = 2ll << 20;

// ---------------------------------------------------------------- errors
static thread_local int g_err = HB_OK;
static thread_local char g_msg[512] = "";

static bool strict_mode() {
    const char* s = getenv("HYDRO_B200_STRICT");
    return s && s[0] == '1';
}

static int set_error(int code, const char* fmt, ...) {
    g_err = code;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_msg, sizeof(g_msg), fmt, ap);
    va_end(ap);
    if (strict_mode()) {
        fprintf(stderr, "hydro_b200: error %d: %s\n", code, g_msg);
        abort();
    }
    return code;
}

#define HB_CU(call)                                                                      \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess)                                                           \
            return set_error(e_ == cudaErrorMemoryAllocation ? HB_ERR_NOMEM : HB_ERR_CUDA, \
                             "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_),     \
                             __FILE__, __LINE__);                                        \
    } while (0)

// Records an error from another translation unit of the library.
int hb_record_error(int code, const char* msg) { return set_error(code, "%s", msg); }

extern "C" int hydro_b200_last_error(void) { return g_err; }
extern "C" const char* hydro_b200_last_error_message(void) { return g_msg; }
extern "C" void hydro_b200_clear_error(void) {
    g_err = HB_OK;
    g_msg[0] = 0;
}

// ---------------------------------------------------------------- domain
struct HostPage;  // see take_host_pair
struct hb_domain {
    int nx = 0, ny = 0, nxt = 0, nyt = 0;
    long long vs = 0;
    size_t nelem = 0;                  // 4 * nxt * nyt
    double* A = nullptr;               // resident state
    double* B = nullptr;               // scratch: output of the first sweep of a step
    unsigned long long* cour = nullptr;  // [2 * kCourSlots] Courant maxima (bit patterns)
    unsigned long long* host_max = nullptr;  // a pair of mapped host memory, or null
    HostPage* host_page = nullptr;           // the page it lies in
    DevClock* clk = nullptr;
    int2* todo = nullptr;              // the cooperative sweeps' window list
    unsigned* todo_count = nullptr;    // its length, ticket and claims (SweepArgs)
    double* dts = nullptr;
    int ndts = 0;
    cudaStream_t stream = nullptr;
    int device = 0;
    Phys P{};
    double courant_factor = 0.0;
    int bnd_left = 1, bnd_right = 1, bnd_down = 1, bnd_up = 1;
    int sm_count = 0;  // cudaDevAttrMultiProcessorCount, read in domain_alloc
    int precision = HB_PREC_FP64;
    // Sweep kernel (HB_KERNEL_*) per [precision][direction]; set in domain_alloc.
    int kern[3][3] = {{0, HB_KERNEL_WARP, HB_KERNEL_MARCH},
                      {0, HB_KERNEL_WARP, HB_KERNEL_MARCH},
                      {0, HB_KERNEL_WARP, HB_KERNEL_MARCH}};
    bool mixed_auto[3] = {false, true, true};  // kern[HB_PREC_MIXED][dir] is the default's choice
    int seg[3][3] = {{0, 64, 64}, {0, 64, 64}, {0, 64, 64}};  // [precision][direction]
    bool cour_valid = false;  // cour holds the maxima of the current state
    int h_nstep = 0;          // host view of the clock's nstep (parity of launches)
    bool h_ahead = false;     // steps were launched that the clock may have stopped before
    long long launches = 0;
    // Optional event timing of every sweep launch (hydro_b200_domain_profile).
    bool prof = false;
    std::vector<cudaEvent_t> ev_pool;    // free events
    std::vector<cudaEvent_t> ev_pending; // start/end pairs, sweep direction in ev_dir
    std::vector<int> ev_dir;
    double prof_ms[2] = {0.0, 0.0};
    long long prof_n[2] = {0, 0};
    unsigned char* b64 = nullptr;  // VTK output text of one variable (hb_output.cu)
    size_t b64_cap = 0;
    // The launch-only driver replays an even + odd step pair from a CUDA
    // graph; pair_key holds what the captured launches were built from.
    cudaGraphExec_t pair_exec = nullptr;
    std::vector<unsigned char> pair_key;
};

static int validate(const hydroparam_t* H) {
    if (!H) return set_error(HB_ERR_ARG, "null hydroparam_t");
    if (H->nvar != 4)
        return set_error(HB_ERR_ARG, "nvar=%d: only the reference's 4 variables are supported",
                         H->nvar);
    if (H->nx < 3 || H->ny < 3)
        return set_error(HB_ERR_ARG, "grid %dx%d: nx and ny must be >= 3", H->nx, H->ny);
    if (((long long)H->nx + 4) * ((long long)H->ny + 4) > (1ll << 31))
        return set_error(HB_ERR_ARG, "grid too large for 32-bit line indices");
    if ((H->nxt && H->nxt != H->nx + 4) || (H->nyt && H->nyt != H->ny + 4))
        return set_error(HB_ERR_ARG, "nxt/nyt (%d,%d) must be nx+4, ny+4", H->nxt, H->nyt);
    if (H->scheme < 1 || H->scheme > 3)
        return set_error(HB_ERR_ARG, "scheme=%d: expected 1 (muscl), 2 (plmde) or 3 (collela)",
                         H->scheme);
    if (!(H->dx > 0.0)) return set_error(HB_ERR_ARG, "dx must be > 0");
    if (H->niter_riemann < 0) return set_error(HB_ERR_ARG, "niter_riemann < 0");
    return HB_OK;
}

// Constants of the run, with the reference's formulas (see hb_stages.cuh).
static void load_params(hb_domain* d, const hydroparam_t* H) {
    Phys& P = d->P;
    P.gamma = H->gamma;
    P.gm1 = H->gamma - 1.0;
    P.smallr = H->smallr;
    P.smallc = H->smallc;
    P.smallp = (H->smallc * H->smallc) / H->gamma;
    P.gamma6 = (H->gamma + 1.0) / (2.0 * H->gamma);
    P.smallpp = H->smallr * P.smallp;
    P.entho = 1.0 / (H->gamma - 1.0);
    P.slope_type = H->slope_type;
    P.dx = H->dx;
    P.niter = H->niter_riemann;
    P.iorder = H->iorder;
    P.scheme = H->scheme;
    P.unit_slope = (H->slope_type == 1.0) ? 1 : 0;
    d->courant_factor = H->courant_factor;
    d->bnd_left = H->boundary_left;
    d->bnd_right = H->boundary_right;
    d->bnd_down = H->boundary_down;
    d->bnd_up = H->boundary_up;
}

static void give_host_pair(hb_domain* d);  // beside domain_alloc

extern "C" void hydro_b200_domain_destroy(hb_domain* d) {
    if (!d) return;
    if (d->stream) cudaStreamSynchronize(d->stream);
    for (cudaEvent_t e : d->ev_pool) cudaEventDestroy(e);
    for (cudaEvent_t e : d->ev_pending) cudaEventDestroy(e);
    cudaFree(d->A);
    cudaFree(d->B);  // and the records behind it (domain_alloc)
    give_host_pair(d);
    cudaFree(d->dts);
    cudaFree(d->b64);
    if (d->pair_exec) cudaGraphExecDestroy(d->pair_exec);
    if (d->stream) cudaStreamDestroy(d->stream);
    delete d;
}

// Segment length of a sweep: the grid has ceil(nlines/64) x ceil(nl/seg) CTAs,
// each marching one segment plus a 4-cell halo.  Measured on B200:
//  - a grid with fewer CTAs than resident slots runs them all at once, so its
//    time is one segment's: shorter segments (down to 8 cells) help until the
//    grid fills a wave (512^2 FP64 y sweep: 0.41 ms at seg 64, 0.09 ms at 8);
//  - otherwise the length that fills whole waves best, weighed against the
//    halo (about 1.6/seg of the work), capped at `cap`: the FP64 y sweep runs
//    faster with several waves of ~32-cell segments than with one wave of
//    long ones (4096^2: 1.43 against 1.49 ms; 8192^2: 5.41 against 5.61 ms).
static int choose_seg(int nlines, int nl, int slots, int cap) {
    const long long groups = (nlines + hb::kSweepThreads - 1) / hb::kSweepThreads;
    auto ctas = [&](int seg) { return groups * ((nl + seg - 1) / seg); };
    if (ctas(24) < slots) {
        int seg = 24;
        while (seg > 8 && ctas(seg) < slots) seg -= 2;
        return seg;
    }
    int best = 24;
    double best_score = -1.0;
    // Even lengths keep every thread's first cell 16-byte aligned for the x
    // sweep's vector loads.
    for (int seg = 24; seg <= nl + 1 && seg <= 8192; seg += 2) {
        const long long n = ctas(seg);
        const long long waves = (n + slots - 1) / slots;
        const double fill = (double)n / (double)(waves * slots);
        const double score = fill / (1.0 + 1.6 / seg);
        if (score > best_score + 1e-9) {
            best_score = score;
            best = seg;
        }
    }
    return best < cap ? best : cap;
}

// The measured default sweep kernel of a grid (per-sweep times on B200, FP64, us):
//
//   cells      input                   x: warp  coop      y: warp  coop   march
//   4096^2     centred blast              300   209         315     223     447
//   4096^2     energy noise              1032  1023         993    1005    1130
//   2048^2     centred blast               82    71          84      71     170
//   2048^2     energy noise               277   280         261     275     300
//   3001x777   centred blast               48    50          51      58     127
//   3001x777   energy noise               156   163         154     173     232
//   1024^2     centred blast               24    32          23      41      79
//   1024^2     energy noise                83    93          75      91     105
//   FMA tier:
//   2048^2     smooth flow                173   160         174     170
//   3001x777   smooth flow / at rest    99/47 95/43      102/53  107/53
//   1448^2     smooth flow / at rest    90/44 88/40       91/46   96/43
//   1024^2     smooth flow / at rest    49/22 53/27       50/23   58/35
//
//  - FP64 and FMA: the cooperative windows from kCoopMinCells (FMA:
//    kCoopMinCellsFma) cells, where their two launches and the list cost less
//    than they spread; the warp windows below.
//  - mixed x: the warp window, mixed y: the marcher (small grids: hb_mixed.cu).
static int default_kernel(const hb_domain* d, int prec, int dir) {
    if (prec == HB_PREC_MIXED) return dir == 1 ? HB_KERNEL_WARP : HB_KERNEL_MARCH;
    const long long cells = (long long)d->nx * d->ny;
    return cells >= (prec == HB_PREC_FP64 ? kCoopMinCells : kCoopMinCellsFma) ? HB_KERNEL_COOP : HB_KERNEL_WARP;
}

// Two 8-byte words of mapped host memory per domain, from a page that the
// context keeps: a pinned page taken and freed with each domain would cost
// 1.2 + 0.5 ms where nothing else holds pinned memory.  A page is gone with its
// context (a reset of the device), so pages go by the context's id, which the
// process never uses twice; what stays of a lost page is its record.  None left
// (or no page, or no id): the domain copies its Courant slots instead.
static constexpr int kHostPairs = 256;
struct HostPage {
    unsigned long long context;
    unsigned long long* words;
    bool used[kHostPairs];
};
static std::mutex g_page_mu;
static std::vector<HostPage*> g_pages;
static void* driver_entry(const char* name) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPointByVersion(name, &f, 12000, cudaEnableDefault, &r) != cudaSuccess)
        cudaGetLastError();
    return f;
}
static bool context_id(unsigned long long* id) {
    // The driver's functions, looked up once.
    static const auto current = reinterpret_cast<CUresult (*)(CUcontext*)>(driver_entry("cuCtxGetCurrent"));
    static const auto get_id =
        reinterpret_cast<CUresult (*)(CUcontext, unsigned long long*)>(driver_entry("cuCtxGetId"));
    CUcontext c = nullptr;
    return current && get_id && current(&c) == CUDA_SUCCESS && c && get_id(c, id) == CUDA_SUCCESS;
}
static void take_host_pair(hb_domain* d) {
    unsigned long long id = 0;
    if (!context_id(&id)) return;
    std::lock_guard<std::mutex> lk(g_page_mu);
    HostPage* page = nullptr;
    for (HostPage* p : g_pages)
        if (p->context == id) page = p;
    if (!page) {
        unsigned long long* words = nullptr;
        if (cudaHostAlloc(&words, kHostPairs * 2 * sizeof(*words), cudaHostAllocMapped) !=
            cudaSuccess) {
            cudaGetLastError();
            return;
        }
        page = new HostPage{id, words, {}};
        g_pages.push_back(page);
    }
    for (int i = 0; i < kHostPairs; i++)
        if (!page->used[i]) {
            page->used[i] = true;
            d->host_page = page;
            d->host_max = page->words + 2 * i;
            return;
        }
}
static void give_host_pair(hb_domain* d) {
    if (!d->host_page) return;
    std::lock_guard<std::mutex> lk(g_page_mu);
    d->host_page->used[(d->host_max - d->host_page->words) / 2] = false;
}

static int domain_alloc(hb_domain* d) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        return set_error(HB_ERR_NODEV, "no CUDA device visible");
    HB_CU(cudaGetDevice(&d->device));
    HB_CU(cudaDeviceGetAttribute(&d->sm_count, cudaDevAttrMultiProcessorCount, d->device));
    for (int dir = 1; dir <= 2; dir++) {
        for (int prec = 0; prec < 3; prec++) {
            const int per_sm = prec == HB_PREC_FP64    ? hb::sweep_blocks_per_sm(dir, d->P.unit_slope != 0)
                               : prec == HB_PREC_MIXED ? hb::sweep_mixed_blocks_per_sm(dir)
                                                       : hb::sweep_fast_blocks_per_sm(dir);
            const int slots = d->sm_count * per_sm;
            const int cap = (prec != HB_PREC_MIXED && dir == 2) ? 32 : 1 << 30;
            d->seg[prec][dir] = dir == 1 ? choose_seg(d->ny, d->nx, slots, cap)
                                         : choose_seg(d->nx, d->ny, slots, cap);
        }
    }
    for (int prec = 0; prec < 3; prec++)
        for (int dir = 1; dir <= 2; dir++) d->kern[prec][dir] = default_kernel(d, prec, dir);
    HB_CU(cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking));
    HB_CU(cudaMalloc(&d->A, d->nelem * sizeof(double)));
    // The small records and the window list lie behind the scratch, 256 bytes
    // apart or more (a list of its own is another 0.3 ms of allocation at 4096^2).
    const size_t small_at = (d->nelem * sizeof(double) + 255) / 256 * 256;
    const size_t clk_at = (kCourBytes + 255) / 256 * 256;
    const size_t count_at = clk_at + (sizeof(DevClock) + 255) / 256 * 256, todo_at = count_at + 256;
    HB_CU(cudaMalloc(&d->B,
                     small_at + todo_at + hb::coop_list_size(d->nx, d->ny) * sizeof(int2)));
    char* small = reinterpret_cast<char*>(d->B) + small_at;
    d->cour = reinterpret_cast<unsigned long long*>(small);
    d->clk = reinterpret_cast<DevClock*>(small + clk_at);
    d->todo_count = reinterpret_cast<unsigned*>(small + count_at);
    d->todo = reinterpret_cast<int2*>(small + todo_at);
    HB_CU(cudaMemsetAsync(small, 0, todo_at, d->stream));
    take_host_pair(d);
    return HB_OK;
}

extern "C" hb_domain* hydro_b200_domain_create(const hydroparam_t* H) {
    if (validate(H) != HB_OK) return nullptr;
    hb_domain* d = new hb_domain();
    d->nx = H->nx;
    d->ny = H->ny;
    d->nxt = H->nx + 4;
    d->nyt = H->ny + 4;
    d->vs = (long long)d->nxt * d->nyt;
    d->nelem = (size_t)4 * d->vs;
    load_params(d, H);
    if (domain_alloc(d) != HB_OK) {
        hydro_b200_domain_destroy(d);
        return nullptr;
    }
    return d;
}

extern "C" double* hydro_b200_domain_state(hb_domain* d) { return d ? d->A : nullptr; }
extern "C" void* hydro_b200_domain_stream(hb_domain* d) { return d ? (void*)d->stream : nullptr; }
extern "C" long long hydro_b200_domain_launch_count(hb_domain* d) { return d ? d->launches : 0; }

extern "C" int hydro_b200_domain_upload(hb_domain* d, const double* host) {
    if (!d || !host) return set_error(HB_ERR_ARG, "null domain or buffer");
    HB_CU(cudaMemcpyAsync(d->A, host, d->nelem * sizeof(double), cudaMemcpyHostToDevice,
                          d->stream));
    d->cour_valid = false;
    return HB_OK;
}

extern "C" int hydro_b200_domain_download(hb_domain* d, double* host) {
    if (!d || !host) return set_error(HB_ERR_ARG, "null domain or buffer");
    HB_CU(cudaMemcpyAsync(host, d->A, d->nelem * sizeof(double), cudaMemcpyDeviceToHost,
                          d->stream));
    return HB_OK;
}

extern "C" int hydro_b200_domain_synchronize(hb_domain* d) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    HB_CU(cudaStreamSynchronize(d->stream));
    if (d->precision == HB_PREC_MIXED && d->kern[HB_PREC_MIXED][1] == HB_KERNEL_BULK &&
        hb::mixed_stage_wait_timeouts(true) != 0)
        return set_error(HB_ERR_CUDA, "a staged bulk copy of the mixed x sweep did not complete");
    return HB_OK;
}


static SweepArgs sweep_args(hb_domain* d, int dir, const double* in, double* out,
                            const DevClock* clk, double dt, unsigned long long* cour) {
    SweepArgs a;
    a.in = in;
    a.resid = d->A;
    a.out = out;
    a.gout = d->A;
    a.clk = clk;
    a.odd = 0;
    a.dt = dt;
    a.courant = cour;
    a.nx = d->nx;
    a.ny = d->ny;
    a.nxt = d->nxt;
    a.nyt = d->nyt;
    a.vs = d->vs;
    if (dir == 1) {
        a.bnd_lo = d->bnd_left;
        a.bnd_hi = d->bnd_right;
        a.nlines = d->ny;
        a.n = d->nxt;
    } else {
        a.bnd_lo = d->bnd_down;
        a.bnd_hi = d->bnd_up;
        a.nlines = d->nx;
        a.n = d->nyt;
    }
    a.seg = d->seg[d->precision][dir];
    a.w_lo = 0;
    a.w_hi = hb::kWholeLine;
    a.one_cell = d->precision == HB_PREC_MIXED && d->mixed_auto[dir] &&
                 (long long)d->nx * d->ny <= hb::kOneCellMixedMaxCells;
    a.todo = d->todo;
    a.todo_count = d->todo_count;
    a.empty = nullptr;
    a.dependent = 0;
    return a;
}

static cudaEvent_t take_event(hb_domain* d) {
    if (!d->ev_pool.empty()) {
        cudaEvent_t e = d->ev_pool.back();
        d->ev_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}

// Kernels of one sweep: the cooperative windows take two.
static int sweep_kernels(const hb_domain* d, int dir) {
    const int kern = d->kern[d->precision][dir];
    return kern == HB_KERNEL_COOP || kern == HB_KERNEL_COOP8 ? 2 : 1;
}

static int launch_sweep_timed(hb_domain* d, int dir, const SweepArgs& a) {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (d->prof) {
        e0 = take_event(d);
        e1 = take_event(d);
        HB_CU(cudaEventRecord(e0, d->stream));
    }
    const int kern = d->kern[d->precision][dir];
    if (d->precision == HB_PREC_FP64_FMA) {
        HB_CU(hb::launch_sweep_fast(dir, kern, a, d->P, d->stream));
    } else if (d->precision == HB_PREC_MIXED) {
        if (kern == HB_KERNEL_COOP || kern == HB_KERNEL_COOP8)
            HB_CU(hb::launch_coop_mixed(dir, kern == HB_KERNEL_COOP8 ? 8 : 4, a, d->P, d->stream));
        else if ((kern == HB_KERNEL_WARP || kern == HB_KERNEL_BULK) && dir == 1)
            HB_CU(hb::launch_xcell_mixed(a, d->P, d->stream, kern == HB_KERNEL_BULK));
        else
            HB_CU(hb::launch_sweep_mixed(dir, a, d->P, d->stream));
    } else {
        if (kern == HB_KERNEL_COOP || kern == HB_KERNEL_COOP8)
            HB_CU(hb::launch_coop(dir, kern == HB_KERNEL_COOP8 ? 8 : 4, a, d->P, d->stream));
        else if (kern == HB_KERNEL_WARP)
            HB_CU(dir == 1 ? hb::launch_xcell(a, d->P, d->stream)
                           : hb::launch_ycell(a, d->P, d->stream));
        else
            HB_CU(hb::launch_sweep(dir, a, d->P, d->stream));
    }
    d->launches += sweep_kernels(d, dir);
    if (d->prof) {
        HB_CU(cudaEventRecord(e1, d->stream));
        d->ev_pending.push_back(e0);
        d->ev_pending.push_back(e1);
        d->ev_dir.push_back(dir);
    }
    return HB_OK;
}

// hydro_godunov.c:70-139: first sweep A -> B (ghosts of its direction written
// to A), second sweep B -> A (ghosts of the second direction written to A).
// With fuse, the second sweep also reduces the Courant maxima of the result
// into accumulators that are empty: under a clock its kernels empty them before
// a step that runs (and leave them alone before one that does not), else the
// first sweep empties them.
static int domain_step(hb_domain* d, int idim, double dt, const DevClock* clk, bool fuse) {
    const int first = (idim == 1) ? 1 : 2;
    const int second = 3 - first;
    d->cour_valid = false;  // also when a launch is refused
    SweepArgs a1 = sweep_args(d, first, d->A, d->B, clk, dt, nullptr);
    if (fuse && !clk) a1.empty = d->cour;
    a1.odd = idim == 2;  // under a clock, odd steps sweep y first
    int rc = launch_sweep_timed(d, first, a1);
    if (rc) return rc;
    SweepArgs a2 = sweep_args(d, second, d->B, d->A, clk, dt, fuse ? d->cour : nullptr);
    a2.odd = a1.odd;
    rc = launch_sweep_timed(d, second, a2);
    if (rc) return rc;
    d->cour_valid = fuse;
    return HB_OK;
}

extern "C" int hydro_b200_domain_godunov(hb_domain* d, int idim, double dt, int fuse_courant) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (idim != 1 && idim != 2) return set_error(HB_ERR_ARG, "idim=%d: expected 1 or 2", idim);
    return domain_step(d, idim, dt, nullptr, fuse_courant != 0);
}

// One sweep of a step, for drivers that act between the two sweeps (a domain
// split exchanging halos, mpibounds.c:165-310 called from make_boundary.c:48).
// Stage 0 is the step's first sweep (A -> B), stage 1 the second (B -> A).
extern "C" int hydro_b200_domain_sweep(hb_domain* d, int stage, int idim, double dt,
                                       int fuse_courant) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (idim != 1 && idim != 2) return set_error(HB_ERR_ARG, "idim=%d: expected 1 or 2", idim);
    if (stage != 0 && stage != 1) return set_error(HB_ERR_ARG, "stage=%d: expected 0 or 1", stage);
    if (stage == 0 && fuse_courant)
        return set_error(HB_ERR_ARG, "the Courant reduction fuses into the second sweep only");
    d->cour_valid = false;
    if (fuse_courant) HB_CU(cudaMemsetAsync(d->cour, 0, kCourBytes, d->stream));
    SweepArgs a = stage == 0 ? sweep_args(d, idim, d->A, d->B, nullptr, dt, nullptr)
                             : sweep_args(d, idim, d->B, d->A, nullptr, dt,
                                          fuse_courant ? d->cour : nullptr);
    const int rc = launch_sweep_timed(d, idim, a);
    if (rc) return rc;
    d->cour_valid = stage == 1 && fuse_courant;
    return HB_OK;
}

// Window (segment) geometry of the domain's sweep kernel in direction dir:
// `total` windows per line, of which [lo, hi) read no ghost cell.  Window w
// of the cell-window kernels outputs [W w, W w + W) and reads two cells more
// on each side; segment w of the marching kernels outputs
// [2 + seg w, 2 + seg (w + 1)) and reads the same margins.
static void window_bounds(const hb_domain* d, int dir, int* total, int* lo, int* hi) {
    const int n = dir == 1 ? d->nxt : d->nyt;
    const int kern = d->kern[d->precision][dir];
    if (kern == HB_KERNEL_MARCH) {
        const int seg = d->seg[d->precision][dir];
        *total = (n - 4 + seg - 1) / seg;
        *lo = 1;
        *hi = (n - 6) / seg;
    } else {
        int W = hb::kCellWarpOut;
        if (kern == HB_KERNEL_COOP) W = hb::coop_outputs(dir, 4);
        if (kern == HB_KERNEL_COOP8) W = hb::coop_outputs(dir, 8);
        if ((kern == HB_KERNEL_WARP || kern == HB_KERNEL_BULK) && dir == 1 &&
            d->precision == HB_PREC_MIXED)
            W = hb::kCellWarpOut2;
        *total = (n - 2 + W - 1) / W;
        *lo = 1;
        *hi = (n - 4) / W;
    }
    if (*hi > *total) *hi = *total;
    if (*hi < *lo) *hi = *lo;  // no ghost-free window: part 1 is empty
}

// One part of a sweep (see include/hydro_b200.h): part 1 the ghost-free
// windows, part 2 the others, part 0 all of them.
extern "C" int hydro_b200_domain_sweep_part(hb_domain* d, int stage, int idim, double dt,
                                            int fuse_courant, int part) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (part == 0) return hydro_b200_domain_sweep(d, stage, idim, dt, fuse_courant);
    if (idim != 1 && idim != 2) return set_error(HB_ERR_ARG, "idim=%d: expected 1 or 2", idim);
    if (stage != 0 && stage != 1) return set_error(HB_ERR_ARG, "stage=%d: expected 0 or 1", stage);
    if (part != 1 && part != 2) return set_error(HB_ERR_ARG, "part=%d: expected 0, 1 or 2", part);
    if (stage == 0 && fuse_courant)
        return set_error(HB_ERR_ARG, "the Courant reduction fuses into the second sweep only");
    d->cour_valid = false;
    if (fuse_courant && part == 1) HB_CU(cudaMemsetAsync(d->cour, 0, kCourBytes, d->stream));
    SweepArgs a = stage == 0 ? sweep_args(d, idim, d->A, d->B, nullptr, dt, nullptr)
                             : sweep_args(d, idim, d->B, d->A, nullptr, dt,
                                          fuse_courant ? d->cour : nullptr);
    int total, lo, hi;
    window_bounds(d, idim, &total, &lo, &hi);
    const int ranges[2][2] = {{part == 1 ? lo : 0, part == 1 ? hi : lo}, {hi, total}};
    for (int r = 0; r < (part == 1 ? 1 : 2); r++) {
        if (ranges[r][1] <= ranges[r][0]) continue;
        a.w_lo = ranges[r][0];
        a.w_hi = ranges[r][1];
        const int rc = launch_sweep_timed(d, idim, a);
        if (rc) return rc;
    }
    d->cour_valid = stage == 1 && fuse_courant && part == 2;
    return HB_OK;
}

static int halo_args(hb_domain* d, int idim, int side, const void* buf) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (idim != 1 && idim != 2) return set_error(HB_ERR_ARG, "idim=%d: expected 1 or 2", idim);
    if (side != 0 && side != 1) return set_error(HB_ERR_ARG, "side=%d: expected 0 or 1", side);
    if (!buf) return set_error(HB_ERR_ARG, "null halo buffer");
    return HB_OK;
}

extern "C" long long hydro_b200_domain_halo_count(hb_domain* d, int idim) {
    if (!d || (idim != 1 && idim != 2)) return 0;
    return 8ll * (idim == 1 ? d->ny : d->nx);
}

extern "C" int hydro_b200_domain_halo_pack(hb_domain* d, int stage, int idim, int side,
                                           double* dst) {
    int rc = halo_args(d, idim, side, dst);
    if (rc) return rc;
    if (stage != 0 && stage != 1) return set_error(HB_ERR_ARG, "stage=%d: expected 0 or 1", stage);
    // Before the first sweep the state is A; before the second, the first
    // sweep's output B holds the interior.
    HB_CU(hb::launch_halo(stage == 0 ? d->A : d->B, dst, 1, idim, side, d->nx, d->ny, d->nxt,
                          d->vs, d->stream));
    d->launches += 1;
    return HB_OK;
}

extern "C" int hydro_b200_domain_halo_unpack(hb_domain* d, int idim, int side,
                                             const double* src) {
    int rc = halo_args(d, idim, side, src);
    if (rc) return rc;
    // Ghost cells of both sweeps are read from A.
    HB_CU(hb::launch_halo(d->A, const_cast<double*>(src), 0, idim, side, d->nx, d->ny, d->nxt,
                          d->vs, d->stream));
    d->launches += 1;
    return HB_OK;
}

// vtkfile.c:262-280 on the device: variable `var` of the interior as floats,
// base64-encoded, into host memory (hydro_b200_vtk_base64_len(nx, ny) bytes).
extern "C" int hydro_b200_domain_vtk_base64(hb_domain* d, int var, char* host_out,
                                            long long cap) {
    if (!d || !host_out) return set_error(HB_ERR_ARG, "null argument");
    if (var < 0 || var > 3) return set_error(HB_ERR_ARG, "var=%d: expected 0..3", var);
    const long long n = hydro_b200_vtk_base64_len(d->nx, d->ny);
    if (cap < n) return set_error(HB_ERR_ARG, "output buffer of %lld bytes < %lld", cap, n);
    if (d->b64_cap < (size_t)n + 16) {
        cudaFree(d->b64);
        d->b64 = nullptr;
        d->b64_cap = 0;
        HB_CU(cudaMalloc(&d->b64, (size_t)n + 16));
        d->b64_cap = (size_t)n + 16;
    }
    HB_CU(hb::launch_vtk_base64(d->A + var * d->vs, d->nx, d->ny, d->nxt, d->b64, d->stream));
    d->launches += 1;
    HB_CU(cudaMemcpyAsync(host_out, d->b64, (size_t)n, cudaMemcpyDeviceToHost, d->stream));
    HB_CU(cudaStreamSynchronize(d->stream));
    return HB_OK;
}

extern "C" int hydro_b200_domain_set_precision(hb_domain* d, int precision) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (precision != HB_PREC_FP64 && precision != HB_PREC_MIXED && precision != HB_PREC_FP64_FMA)
        return set_error(HB_ERR_ARG,
                         "precision=%d: expected HB_PREC_FP64, HB_PREC_MIXED or HB_PREC_FP64_FMA",
                         precision);
    d->precision = precision;
    return HB_OK;
}

extern "C" int hydro_b200_domain_set_xsweep(hb_domain* d, int precision, int mode) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (precision < HB_PREC_FP64 || precision > HB_PREC_FP64_FMA ||
        (mode != HB_XSWEEP_MARCH && mode != HB_XSWEEP_CELL))
        return set_error(HB_ERR_ARG, "precision=%d mode=%d: invalid", precision, mode);
    d->kern[precision][1] = mode == HB_XSWEEP_CELL ? HB_KERNEL_WARP : HB_KERNEL_MARCH;
    if (precision == HB_PREC_MIXED) d->mixed_auto[1] = false;
    return HB_OK;
}

extern "C" int hydro_b200_domain_set_kernel(hb_domain* d, int precision, int idim, int kernel) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (precision < HB_PREC_FP64 || precision > HB_PREC_FP64_FMA || (idim != 1 && idim != 2))
        return set_error(HB_ERR_ARG, "precision=%d idim=%d: invalid", precision, idim);
    const bool by_default = kernel == HB_KERNEL_AUTO;
    if (by_default) kernel = default_kernel(d, precision, idim);
    const bool known = kernel == HB_KERNEL_MARCH || kernel == HB_KERNEL_WARP ||
                       kernel == HB_KERNEL_COOP || kernel == HB_KERNEL_COOP8 ||
                       kernel == HB_KERNEL_BULK;
    // The mixed set's warp window along columns is the default's own, for small
    // grids (sweep_args); bulk staging exists for the mixed x sweep only.
    if (!known || (precision == HB_PREC_MIXED && idim == 2 && kernel == HB_KERNEL_WARP) ||
        (kernel == HB_KERNEL_BULK && (precision != HB_PREC_MIXED || idim != 1)))
        return set_error(HB_ERR_ARG, "kernel=%d: not available for precision %d, idim %d", kernel,
                         precision, idim);
    d->kern[precision][idim] = kernel;
    if (precision == HB_PREC_MIXED) d->mixed_auto[idim] = by_default;
    return HB_OK;
}

extern "C" int hydro_b200_domain_get_kernel(hb_domain* d, int precision, int idim) {
    if (!d || precision < HB_PREC_FP64 || precision > HB_PREC_FP64_FMA ||
        (idim != 1 && idim != 2))
        return set_error(HB_ERR_ARG, "invalid domain, precision or idim"), -1;
    return d->kern[precision][idim];
}

extern "C" int hydro_b200_domain_profile(hb_domain* d, int enable) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    d->prof = enable != 0;
    return HB_OK;
}

// Waits for the recorded sweeps and returns the accumulated time (ms) and
// launch count of the x (index 0) and y (index 1) sweeps; reset clears them.
extern "C" int hydro_b200_domain_profile_read(hb_domain* d, double* ms, long long* count,
                                              int reset) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    HB_CU(cudaStreamSynchronize(d->stream));
    for (size_t i = 0; i < d->ev_dir.size(); i++) {
        float t = 0.f;
        HB_CU(cudaEventElapsedTime(&t, d->ev_pending[2 * i], d->ev_pending[2 * i + 1]));
        d->prof_ms[d->ev_dir[i] - 1] += t;
        d->prof_n[d->ev_dir[i] - 1] += 1;
    }
    for (cudaEvent_t e : d->ev_pending) d->ev_pool.push_back(e);
    d->ev_pending.clear();
    d->ev_dir.clear();
    if (ms) {
        ms[0] = d->prof_ms[0];
        ms[1] = d->prof_ms[1];
    }
    if (count) {
        count[0] = d->prof_n[0];
        count[1] = d->prof_n[1];
    }
    if (reset) {
        d->prof_ms[0] = d->prof_ms[1] = 0.0;
        d->prof_n[0] = d->prof_n[1] = 0;
    }
    return HB_OK;
}

extern "C" int hydro_b200_domain_make_boundary(hb_domain* d, int idim) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (idim != 1 && idim != 2) return set_error(HB_ERR_ARG, "idim=%d: expected 1 or 2", idim);
    const int lo = idim == 1 ? d->bnd_left : d->bnd_down;
    const int hi = idim == 1 ? d->bnd_right : d->bnd_up;
    HB_CU(hb::launch_boundary(d->A, idim, d->nx, d->ny, d->nxt, d->nyt, d->vs, lo, hi,
                              d->stream));
    d->launches += 1;
    return HB_OK;
}

static int ensure_courant(hb_domain* d) {
    if (d->cour_valid) return HB_OK;
    HB_CU(cudaMemsetAsync(d->cour, 0, kCourBytes, d->stream));
    // The per-cell formula of the domain's precision, as in the fused reduction.
    if (d->precision == HB_PREC_FP64_FMA) {
        HB_CU(hb::launch_courant_fast(d->A, d->nx, d->ny, d->nxt, d->vs, d->P, d->cour,
                                      d->stream));
    } else if (d->precision == HB_PREC_MIXED) {
        HB_CU(hb::launch_courant_mixed(d->A, d->nx, d->ny, d->nxt, d->vs, d->P, d->cour,
                                       d->stream));
    } else {
        HB_CU(hb::launch_courant(d->A, d->nx, d->ny, d->nxt, d->vs, d->P, d->cour, d->stream));
    }
    d->launches += 1;
    d->cour_valid = true;
    return HB_OK;
}

// The maxima of steps launched under the clock are the state's own if the clock
// ran them all: a step that it stopped before reduced nothing, and the accumulators
// may have been emptied for the step before that one.  `nstep` is the clock's.
static void settle_steps(hb_domain* d, int nstep) {
    if (d->h_ahead && nstep != d->h_nstep) d->cour_valid = false;
    d->h_ahead = false;
}
// The same where nothing has read the clock yet; waits for the steps.
static int settle_steps(hb_domain* d) {
    if (!d->h_ahead || !d->cour_valid) return HB_OK;
    int nstep = 0;
    HB_CU(cudaMemcpyAsync(&nstep, &d->clk->nstep, sizeof nstep, cudaMemcpyDeviceToHost,
                          d->stream));
    HB_CU(cudaStreamSynchronize(d->stream));
    settle_steps(d, nstep);
    return HB_OK;
}

extern "C" int hydro_b200_domain_courant(hb_domain* d, double* cx, double* cy) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    int rc = settle_steps(d);
    if (rc) return rc;
    rc = ensure_courant(d);
    if (rc) return rc;
    unsigned long long h[2 * hb::kCourSlots], mx = 0, my = 0;
    int dev = -1;
    if (d->host_max && cudaGetDevice(&dev) == cudaSuccess && dev == d->device) {
        HB_CU(hb::launch_courant_read(d->cour, d->host_max, d->stream));
        d->launches += 1;
        HB_CU(cudaStreamSynchronize(d->stream));
        mx = d->host_max[0];
        my = d->host_max[1];
    } else {  // no pair of mapped memory, or another device is current
        HB_CU(cudaMemcpyAsync(h, d->cour, sizeof(h), cudaMemcpyDeviceToHost, d->stream));
        HB_CU(cudaStreamSynchronize(d->stream));
        for (int s = 0; s < hb::kCourSlots; s++) {
            mx = h[s] > mx ? h[s] : mx;
            my = h[hb::kCourSlots + s] > my ? h[hb::kCourSlots + s] : my;
        }
    }
    double x, y;
    memcpy(&x, &mx, 8);
    memcpy(&y, &my, 8);
    if (cx) *cx = x;
    if (cy) *cy = y;
    return HB_OK;
}

extern "C" int hydro_b200_domain_set_clock(hb_domain* d, double t, int nstep, double dt) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    const int rc = settle_steps(d);  // before the clock is overwritten
    if (rc) return rc;
    DevClock c;
    memset(&c, 0, sizeof(c));
    c.t = t;
    c.dt = dt;
    c.tend = 0.0;
    c.nstep = nstep;
    c.nstep0 = nstep;
    c.nstepmax = nstep;
    c.active = 1;
    c.dts = d->dts;
    c.ndts = d->ndts;
    HB_CU(cudaMemcpyAsync(d->clk, &c, sizeof(c), cudaMemcpyHostToDevice, d->stream));
    HB_CU(cudaStreamSynchronize(d->stream));
    d->h_nstep = nstep;
    d->h_ahead = false;
    return HB_OK;
}

// Reserve the device record for the dt of the next n steps.
static int ensure_dts(hb_domain* d, int n) {
    if (n <= d->ndts) return HB_OK;
    cudaFree(d->dts);
    d->dts = nullptr;
    d->ndts = 0;
    HB_CU(cudaMalloc(&d->dts, (size_t)n * sizeof(double)));
    d->ndts = n;
    return HB_OK;
}

// What the captured step pair's launches are built from: kernel arguments are
// captured by value, so any change here needs a new capture.
static std::vector<unsigned char> pair_key(const hb_domain* d) {
    struct Key {
        Phys P;
        double courant_factor;
        int precision, kern1, kern2, auto1, auto2, seg1, seg2, bnd[4];
    } k;
    memset(&k, 0, sizeof(k));
    k.P = d->P;
    k.courant_factor = d->courant_factor;
    k.precision = d->precision;
    k.kern1 = d->kern[d->precision][1];
    k.kern2 = d->kern[d->precision][2];
    k.auto1 = d->precision == HB_PREC_MIXED && d->mixed_auto[1];
    k.auto2 = d->precision == HB_PREC_MIXED && d->mixed_auto[2];
    k.seg1 = d->seg[d->precision][1];
    k.seg2 = d->seg[d->precision][2];
    k.bnd[0] = d->bnd_left;
    k.bnd[1] = d->bnd_right;
    k.bnd[2] = d->bnd_down;
    k.bnd[3] = d->bnd_up;
    const unsigned char* b = reinterpret_cast<const unsigned char*>(&k);
    return std::vector<unsigned char>(b, b + sizeof(k));
}

// The launches of one even step (x then y) and the odd step after it (y then
// x, Courant maxima fused), behind one clock kernel for both: 5 kernels, two
// more for each pair of cooperative sweeps.  Issued into a capture.
static int issue_pair(hb_domain* d) {
    HB_CU(hb::launch_clock_pair(d->clk, d->cour, d->courant_factor, d->P.dx, d->P.smallc,
                                d->stream));
    for (int odd = 0; odd < 2; odd++) {
        const int rc = domain_step(d, odd ? 2 : 1, 0.0, d->clk, odd == 1);
        if (rc) return rc;
    }
    return HB_OK;
}

static int ensure_pair_graph(hb_domain* d) {
    std::vector<unsigned char> key = pair_key(d);
    if (d->pair_exec && key == d->pair_key) return HB_OK;
    if (d->pair_exec) {
        cudaGraphExecDestroy(d->pair_exec);
        d->pair_exec = nullptr;
    }
    const long long launches = d->launches;
    const bool cour_valid = d->cour_valid;
    HB_CU(cudaStreamBeginCapture(d->stream, cudaStreamCaptureModeThreadLocal));
    const int rc = issue_pair(d);
    cudaGraph_t g = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(d->stream, &g);  // always ends the capture
    d->launches = launches;  // captured launches are counted when replayed
    d->cour_valid = cour_valid;
    if (rc != HB_OK) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (ec != cudaSuccess) return set_error(HB_ERR_CUDA, "step-pair capture: %s", cudaGetErrorString(ec));
    const cudaError_t ei = cudaGraphInstantiate(&d->pair_exec, g, 0);
    cudaGraphDestroy(g);
    if (ei != cudaSuccess) {
        d->pair_exec = nullptr;
        return set_error(HB_ERR_CUDA, "step-pair graph: %s", cudaGetErrorString(ei));
    }
    d->pair_key.swap(key);
    return HB_OK;
}

// Asynchronous.  An even step and the odd one after it are replayed from the
// captured pair: one clock kernel for both, then their four sweeps.  A step by
// itself (the first of an odd count, the last of an even one, or while sweeps are
// timed) is a clock kernel (dt on even steps, stop test), its two sweeps and a
// clock kernel (t += dt, nstep++).  The second sweep of odd steps reduces the
// Courant maxima.
extern "C" int hydro_b200_domain_launch_steps(hb_domain* d, int nsteps, int nstepmax,
                                              double tend) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    // Update the limits in the device clock (fields tend, nstepmax).
    HB_CU(cudaMemcpyAsync((char*)d->clk + offsetof(DevClock, tend), &tend, sizeof(double),
                          cudaMemcpyHostToDevice, d->stream));
    HB_CU(cudaMemcpyAsync((char*)d->clk + offsetof(DevClock, nstepmax), &nstepmax, sizeof(int),
                          cudaMemcpyHostToDevice, d->stream));
    d->h_ahead = d->h_ahead || nsteps > 0;
    for (int s = 0; s < nsteps; s++) {
        const int n = d->h_nstep;
        // An even step with its odd successor: replayed from the captured pair
        // (not while sweeps are being timed one by one).  Steps past the stop
        // condition are no-ops on the device, as when launched one by one.
        if (!d->prof && n % 2 == 0 && nsteps - s >= 2) {
            int rc = ensure_courant(d);  // the first step's dt needs the maxima
            if (rc) return rc;
            rc = ensure_pair_graph(d);
            if (rc) return rc;
            HB_CU(cudaGraphLaunch(d->pair_exec, d->stream));
            d->launches += 1 + 2 * (sweep_kernels(d, 1) + sweep_kernels(d, 2));
            d->h_nstep += 2;
            d->cour_valid = true;  // the odd step fused the maxima of the result
            s++;
            continue;
        }
        if (n % 2 == 0) {
            int rc = ensure_courant(d);
            if (rc) return rc;
        }
        HB_CU(hb::launch_clock_begin(d->clk, d->cour, d->courant_factor, d->P.dx, d->P.smallc,
                                     d->stream));
        int rc = domain_step(d, (n % 2 == 0) ? 1 : 2, 0.0, d->clk, (n % 2) == 1);
        if (rc) return rc;
        HB_CU(hb::launch_clock_end(d->clk, d->stream));
        d->launches += 2;
        d->h_nstep++;
        // clock_begin of an even step consumed (zeroed) the accumulators.
        if (n % 2 == 0) d->cour_valid = false;
    }
    return HB_OK;
}

extern "C" int hydro_b200_domain_get_clock(hb_domain* d, double* t, int* nstep, double* dt) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    DevClock c;
    HB_CU(cudaMemcpyAsync(&c, d->clk, sizeof(c), cudaMemcpyDeviceToHost, d->stream));
    HB_CU(cudaStreamSynchronize(d->stream));
    settle_steps(d, c.nstep);
    if (t) *t = c.t;
    if (nstep) *nstep = c.nstep;
    if (dt) *dt = c.dt;
    return HB_OK;
}

extern "C" int hydro_b200_domain_reserve_dts(hb_domain* d, int n) {
    if (!d) return set_error(HB_ERR_ARG, "null domain");
    if (n < 0) return set_error(HB_ERR_ARG, "n=%d: expected >= 0", n);
    return ensure_dts(d, n);
}

extern "C" int hydro_b200_domain_get_dts(hb_domain* d, double* dts, int n) {
    if (!d || !dts) return set_error(HB_ERR_ARG, "null argument");
    if (n > d->ndts) return set_error(HB_ERR_ARG, "only %d dt records reserved", d->ndts);
    if (n <= 0) return HB_OK;
    HB_CU(cudaMemcpyAsync(dts, d->dts, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost,
                          d->stream));
    HB_CU(cudaStreamSynchronize(d->stream));
    return HB_OK;
}

// ------------------------------------------------- mirror registry (ref ABI)
struct Mirror {
    hb_domain* dom;
};
static std::mutex g_mu;
static std::unordered_map<const void*, Mirror> g_mirrors;

static bool sync_each_call() {
    const char* s = getenv("HYDRO_B200_SYNC");
    return s && s[0] == '1';
}

// Find (or create and upload) the mirror of Hv->uold for the grid of H.
static hb_domain* mirror_for(const hydroparam_t* H, hydrovar_t* Hv) {
    if (!Hv || !Hv->uold) {
        set_error(HB_ERR_ARG, "null hydrovar_t or uold");
        return nullptr;
    }
    if (validate(H) != HB_OK) return nullptr;
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_mirrors.find(Hv->uold);
    if (it != g_mirrors.end()) {
        hb_domain* d = it->second.dom;
        if (d->nx == H->nx && d->ny == H->ny) {
            load_params(d, H);  // H is passed by value on every call: take its constants
            return d;
        }
        hydro_b200_domain_destroy(d);
        g_mirrors.erase(it);
    }
    hb_domain* d = hydro_b200_domain_create(H);
    if (!d) return nullptr;
    const char* prec = getenv("HYDRO_B200_PRECISION");
    if (prec && strcmp(prec, "mixed") == 0) d->precision = HB_PREC_MIXED;
    if (prec && strcmp(prec, "fma") == 0) d->precision = HB_PREC_FP64_FMA;
    const char* xs = getenv("HYDRO_B200_XSWEEP");
    const bool cell = xs && strcmp(xs, "cell") == 0, row = xs && strcmp(xs, "march") == 0;
    if (cell || row) {
        d->kern[0][1] = d->kern[1][1] = cell ? HB_KERNEL_WARP : HB_KERNEL_MARCH;
        d->mixed_auto[1] = false;
    }
    if (hydro_b200_domain_upload(d, Hv->uold) != HB_OK) {
        hydro_b200_domain_destroy(d);
        return nullptr;
    }
    g_mirrors[Hv->uold] = Mirror{d};
    return d;
}

extern "C" void* hydro_b200_mirror_stream(const hydroparam_t* H, hydrovar_t* Hv) {
    hb_domain* d = mirror_for(H, Hv);
    return d ? (void*)d->stream : nullptr;
}

extern "C" int hydro_b200_sync_to_host(const hydroparam_t* H, hydrovar_t* Hv) {
    hb_domain* d = mirror_for(H, Hv);
    if (!d) return g_err;
    int rc = hydro_b200_domain_download(d, Hv->uold);
    if (rc) return rc;
    return hydro_b200_domain_synchronize(d);
}

extern "C" int hydro_b200_sync_to_device(const hydroparam_t* H, hydrovar_t* Hv) {
    hb_domain* d = mirror_for(H, Hv);
    if (!d) return g_err;
    int rc = hydro_b200_domain_upload(d, Hv->uold);
    if (rc) return rc;
    return hydro_b200_domain_synchronize(d);
}

extern "C" int hydro_b200_release(hydrovar_t* Hv) {
    if (!Hv) return set_error(HB_ERR_ARG, "null hydrovar_t");
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_mirrors.find(Hv->uold);
    if (it == g_mirrors.end()) return HB_OK;
    hydro_b200_domain_destroy(it->second.dom);
    g_mirrors.erase(it);
    return HB_OK;
}

// The reference's per-stage timer table (parametres.h:150-165, defined by the
// driver at main.c:34 and printed at main.c:515-530).  Weak: it resolves to
// the driver's table when the library is linked into the reference
// application, and to null in any other process.
extern "C" double functim[] __attribute__((weak));
// Slots of the Timers_t enumeration (parametres.h:150-163) the library fills.
static constexpr int kTimRieman = 6;   // TIM_RIEMAN: the fused sweeps (all stages)
static constexpr int kTimMakbou = 10;  // TIM_MAKBOU: make_boundary on its own

// With the driver's timer table present, the entry points time their kernels
// with CUDA events, wait for them (so that the driver's own clock around the
// next call does not absorb this call's device time) and add the seconds to
// functim[slot], as each reference stage adds its own (e.g. riemann.c:287).
struct StageTimer {
    hb_domain* d;
    int slot;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    StageTimer(hb_domain* dom, int s) : d(dom), slot(s) {
        if (!functim) return;
        e0 = take_event(d);
        e1 = take_event(d);
        if (e0 && e1) cudaEventRecord(e0, d->stream);
    }
    void done() {
        if (!functim || !e0 || !e1) return;
        float ms = 0.f;
        if (cudaEventRecord(e1, d->stream) == cudaSuccess &&
            cudaEventSynchronize(e1) == cudaSuccess &&
            cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess)
            functim[slot] += ms * 1e-3;
        release();
    }
    void release() {
        if (e0) d->ev_pool.push_back(e0);
        if (e1) d->ev_pool.push_back(e1);
        e0 = e1 = nullptr;
    }
    ~StageTimer() { release(); }
};

extern "C" void hydro_godunov(int idim, real_t dt, const hydroparam_t H, hydrovar_t* Hv,
                              hydrowork_t* Hw, hydrovarwork_t* Hvw) {
    (void)Hw;
    (void)Hvw;
    hb_domain* d = mirror_for(&H, Hv);
    if (!d) return;
    if (idim != 1 && idim != 2) {
        set_error(HB_ERR_ARG, "idim=%d: expected 1 or 2", idim);
        return;
    }
    // The reference driver calls compute_deltat right after every idim == 2
    // step (main.c:349-399): reduce the Courant maxima inside its second sweep.
    StageTimer tim(d, kTimRieman);
    if (domain_step(d, idim, dt, nullptr, idim == 2) != HB_OK) return;
    tim.done();
    if (sync_each_call()) {
        if (hydro_b200_domain_download(d, Hv->uold) == HB_OK) hydro_b200_domain_synchronize(d);
    }
}

extern "C" void compute_deltat(real_t* dt, const hydroparam_t H, hydrowork_t* Hw, hydrovar_t* Hv,
                               hydrovarwork_t* Hvw) {
    (void)Hw;
    (void)Hvw;
    if (!dt) {
        set_error(HB_ERR_ARG, "null dt");
        return;
    }
    hb_domain* d = mirror_for(&H, Hv);
    if (!d) return;
    double cx = 0.0, cy = 0.0;
    if (hydro_b200_domain_courant(d, &cx, &cy) != HB_OK) return;
    // compute_deltat.c:73 (MAX of utils.h).
    double m = cy > H.smallc ? cy : H.smallc;
    m = cx > m ? cx : m;
    *dt = H.courant_factor * H.dx / m;
}

extern "C" void make_boundary(int idim, const hydroparam_t H, hydrovar_t* Hv) {
    hb_domain* d = mirror_for(&H, Hv);
    if (!d) return;
    StageTimer tim(d, kTimMakbou);  // make_boundary.c:202
    if (hydro_b200_domain_make_boundary(d, idim) != HB_OK) return;
    tim.done();
    if (sync_each_call()) {
        if (hydro_b200_domain_download(d, Hv->uold) == HB_OK) hydro_b200_domain_synchronize(d);
    }
}

int hb_vtk_write(hb_domain* d, int step, const hydroparam_t* H);  // hb_output.cu

// vtkfile.h: the reference's VTK output, written from the device mirror.
extern "C" void vtkfile(int step, const hydroparam_t H, hydrovar_t* Hv) {
    hb_domain* d = mirror_for(&H, Hv);
    if (!d) return;
    if (hb_vtk_write(d, step, &H) != HB_OK && strict_mode()) abort();
}

extern "C" void compute_deltat_init_mem(const hydroparam_t H, hydrowork_t* Hw,
                                        hydrovarwork_t* Hvw) {
    (void)H;
    if (Hw) memset(Hw, 0, sizeof(*Hw));
    if (Hvw) memset(Hvw, 0, sizeof(*Hvw));
}

extern "C" void compute_deltat_clean_mem(const hydroparam_t H, hydrowork_t* Hw,
                                         hydrovarwork_t* Hvw) {
    (void)H;
    (void)Hw;
    (void)Hvw;
    std::lock_guard<std::mutex> lk(g_mu);
    for (auto& kv : g_mirrors) {
        hb_domain* d = kv.second.dom;
        cudaMemcpyAsync((void*)kv.first, d->A, d->nelem * sizeof(double), cudaMemcpyDeviceToHost,
                        d->stream);
        cudaStreamSynchronize(d->stream);
        hydro_b200_domain_destroy(d);
    }
    g_mirrors.clear();
}

extern "C" int hydro_b200_run(const hydroparam_t* H, hydrovar_t* Hv, int nstepmax, real_t tend,
                              real_t* t, int* nstep, real_t* dt, real_t* dts) {
    if (!t || !nstep || !dt) return set_error(HB_ERR_ARG, "null t/nstep/dt"), -1;
    hb_domain* d = mirror_for(H, Hv);
    if (!d) return -1;
    const int todo = nstepmax - *nstep;
    if (todo <= 0 || !(*t < tend)) return 0;
    if (ensure_dts(d, todo) != HB_OK) return -1;
    if (hydro_b200_domain_set_clock(d, *t, *nstep, *dt) != HB_OK) return -1;
    if (hydro_b200_domain_launch_steps(d, todo, nstepmax, tend) != HB_OK) return -1;
    int n1 = *nstep;
    if (hydro_b200_domain_get_clock(d, t, &n1, dt) != HB_OK) return -1;
    const int done = n1 - *nstep;
    if (dts && done > 0 && hydro_b200_domain_get_dts(d, dts, done) != HB_OK) return -1;
    *nstep = n1;
    // The host's parity view must follow the device clock when it stopped early.
    d->h_nstep = n1;
    d->cour_valid = false;
    return done;
}

extern "C" int hydro_b200_set_device(int device) {
    HB_CU(cudaSetDevice(device));
    return HB_OK;
}

extern "C" const char* hydro_b200_build_info(void) {
    return "hydro_b200: FP64 fused sweeps, sm_100a, --fmad=false, IEEE div/sqrt";
}
