// hb_coop.cuh -- the cooperative line window shared by the sweep kernels.
//
// A CTA of T threads takes R = T / C consecutive cells [c - 2, c + R - 2) of each
// of C neighbouring lines, one cell per thread, and produces the updates of
// the N = R - 4 cells [c, c + N).  The stages exchange neighbours through
// shared memory instead of warp shuffles, so the window's halo costs 4 of R
// threads a line instead of 4 of every warp's 32 (the warp window of
// hb_march.cuh, window_output), and the Riemann problems, the dearest stage,
// are solved once per interface but for two:
//
//   phase 1  load cell k = c - 2 + t / C (fused make_boundary), primitives -> smem
//   phase 2  slope (neighbours from smem) + trace -> qxm (kept), qxp -> smem
//   phase 3  Riemann problem + flux at (k | k + 1) from qxm[k], qxp[k + 1] -> smem
//   phase 4  update of cell k with the fluxes of its two faces; store
//
// Along x a window is one row (C = 1).  Along y it is C = 4 columns, the
// columns of a thread group adjacent and starting at a multiple of 4 cells, so
// that every row of the window is a 32-byte sector when the row pitch allows:
// one column a CTA would fetch and write each sector four times.
//
// A sweep is two launches.  The first (steady_body) looks at every window,
// stores the steady ones (hb_march.cuh) and lists the others; it carries no
// stage, so its many light warps keep the memory busy where the gas is at
// rest.  The second (coop_list_body) has one wave of resident CTAs, which take
// the listed windows in turn and sweep them software-pipelined: the work is
// spread evenly however few windows are left.
//
// Measured (4096^2, FP64, x / y, us): where the gas is at rest 205 / 214, the
// copy of the state at 5.2 TB/s, against 705 / 735 when every window went
// through the stages; where every interface iterates 1025 / 1016, bound by
// FP64 (58%) and instruction issue (70%).  One launch that did both kept its
// registers for the stages while it copied, 4 warps in 10 resident, and took
// 290 / 340.
//
// Every cell gets the same stage calls on the same inputs as in the marching
// and warp-window kernels, so the FP64 stage set gives the same bits.
#pragma once

#include "hb_march.cuh"

namespace hb {

// Shared memory of one window, structure of arrays (one 8- or 4-byte element
// per thread and variable: conflict-free accesses).
template <class S, int T>
struct CoopSmem {
    using Real = typename S::Real;
    Real q[4][T];    // primitives
    Real xp[4][T];   // qxp
    double f[4][T];  // flux at (k | k + 1)
};

template <class S, int T>
__device__ __forceinline__ void coop_put(typename S::Real (*dst)[T], int t,
                                         const typename S::Prim& q) {
    dst[0][t] = q.r;
    dst[1][t] = q.u;
    dst[2][t] = q.v;
    dst[3][t] = q.p;
}

template <class S, int T>
__device__ __forceinline__ typename S::Prim coop_get(const typename S::Real (*src)[T], int t) {
    return typename S::Prim{src[0][t], src[1][t], src[2][t], src[3][t]};
}

// Windows of a launch: those of [w_lo, w_hi) on every line (group of C lines).
template <int DIR, int T, int C>
struct CoopGrid {
    static constexpr int R = T / C, N = R - 4;
    int groups, nwin;  // line groups, windows per line
    __host__ __device__ __forceinline__ CoopGrid(const SweepArgs& a) {
        groups = C == 1 ? a.nlines : (a.nlines + 2 + C - 1) / C;
        const int total = (a.n - 2 + N - 1) / N, hi = a.w_hi < total ? a.w_hi : total;
        nwin = hi > a.w_lo ? hi - a.w_lo : 0;
    }
    __host__ __device__ __forceinline__ int windows() const { return groups * nwin; }
};

// The outputs of window `win` of line `line` are [win * N, win * N + N) n
// [2, n - 2).  All threads of the CTA must call this (it has CTA barriers);
// `active` false makes a thread take part in the barriers only.  Warps whose
// cells all lie past the line's end skip the arithmetic.  Accumulates the
// fused Courant maxima of its outputs into cx, cy.
// `staged`: the window's interior cells are already in the stage (thread t's
// cell in staged[v][t], coop_stage_issue), else they are loaded here.
template <class S, int DIR, int T, int C>
__device__ __forceinline__ void coop_window(const SweepArgs& a, const typename S::Consts& Cs,
                                            int line, int win, double dtdx, bool active,
                                            double& cx, double& cy, CoopSmem<S, T>& sm,
                                            const double (*staged)[T]) {
    using Prim = typename S::Prim;
    using Flux = typename S::Flux;
    constexpr int R = T / C, N = R - 4;
    const int t = threadIdx.x, r = t / C;
    const int c = win * N;                          // first output cell of the window
    const int k = c - 2 + r;                        // this thread's cell
    // Threads whose cell is past n + 1 feed nothing that is stored (the last
    // output cell n - 3 needs cells up to n - 1, traced from up to n): whole
    // warps of them skip the arithmetic of a short last window.
    const bool work = active && (c - 2 + (t & ~31) / C) <= a.n;
    const LineGeom<DIR> g(a, line);
    const typename S::TraceK K = S::trace_constants(Cs, dtdx);

    Cons u{1.0, 0.0, 0.0, 1.0};
    Prim q = S::zero_prim();
    typename S::Sound cs = S::zero_sound();
    if (work) {
        constexpr int mn = Slots<DIR>::mn, mt = Slots<DIR>::mt;
        if (staged && k >= 2 && k < a.n - 2)
            u = Cons{staged[0][t], staged[mn][t], staged[mt][t], staged[3][t]};
        else if (k >= 0 && k < a.n)
            u = load_cell<DIR>(a, g, k);
        S::prim(Cs, u, q, cs);
        coop_put<S, T>(sm.q, t, q);
    }
    __syncthreads();
    Prim xm = S::zero_prim();
    if (work) {
        const Prim qm = r > 0 ? coop_get<S, T>(sm.q, t - C) : q;
        const Prim qp = r < R - 1 ? coop_get<S, T>(sm.q, t + C) : q;
        Prim dq = S::zero_prim();
        if (S::second_order(Cs)) S::slope4(Cs, qm, q, qp, dq);
        Prim xp;
        S::trace(K, q, dq, cs, xm, xp);
        coop_put<S, T>(sm.xp, t, xp);
    }
    __syncthreads();
    Flux f = S::zero_flux();
    if (work) {
        const Prim xpn = r < R - 1 ? coop_get<S, T>(sm.xp, t + C) : xm;
        f = S::riemann(Cs, xm, xpn);                // interface (k | k + 1)
        sm.f[0][t] = f.d;
        sm.f[1][t] = f.mn;
        sm.f[2][t] = f.mt;
        sm.f[3][t] = f.e;
    }
    __syncthreads();
    if (work && r >= 2 && r < 2 + N && k >= 2 && k < a.n - 2) {
        const Flux fl{sm.f[0][t - C], sm.f[1][t - C], sm.f[2][t - C], sm.f[3][t - C]};
        const Cons o = S::update(u, fl, f, dtdx);
        store_cell<DIR>(a, g, k, o);
        if (a.courant) take_courant<DIR, S>(Cs, o, cx, cy);
    }
}

// Copies thread t's interior cell of window `win` into stage[v][t] with
// cp.async (one commit group; empty for a ghost or out-of-line cell).
template <int DIR, int T, int C>
__device__ __forceinline__ void coop_stage_issue(const SweepArgs& a, const LineGeom<DIR>& g,
                                                 bool active, int win, double (*stage)[T]) {
    constexpr int N = T / C - 4;
    const int t = threadIdx.x;
    const int k = win * N - 2 + t / C;
    if (active && k >= 2 && k < a.n - 2) {
        const double* p = a.in + g.at(k);
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(&stage[v][t]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst),
                         "l"(p + v * a.vs)
                         : "memory");
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// The first launch.  A few densities of each window are sampled first, so that
// where nothing is uniform a warp pays one round trip to memory; windows whose
// samples agree are loaded whole (16 loads a lane in flight) and stored if
// steady.  The others go to the list, in one claim per warp.
constexpr int kLookThreads = 256;
constexpr int kLookLoads = 4;

// Appends the window (line, win) of each lane with `add` to the list.
__device__ __forceinline__ void list_windows(const SweepArgs& a, bool add, int line, int win) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, add);
    if (m == 0u) return;
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(a.todo_count, (unsigned)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (add) a.todo[at + __popc(m & ((1u << lane) - 1u))] = make_int2(line, win);
}

// Along x: a warp looks at kLookRow windows of the numbering (row by row) in
// turn, the cells of a window across its lanes.
constexpr int kLookRow = 8;
template <class S, int T>
__device__ __forceinline__ void look_rows(const SweepArgs& a, const Phys& P,
                                          const typename S::Consts& Cs, int warp, double& cx,
                                          double& cy) {
    constexpr int R = T, N = R - 4, Q = T / 32;
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const CoopGrid<1, T, 1> grid(a);
    // Lane i < kLookRow holds window i's row and number, lanes 4i .. 4i+3 sample it.
    const int id = warp * kLookRow + (lane & (kLookRow - 1));
    const bool have = id < grid.windows();
    const int row = have ? id / grid.nwin : 0, win = a.w_lo + (have ? id - row * grid.nwin : 0);
    const int srow = __shfl_sync(kAll, row, lane >> 2), swin = __shfl_sync(kAll, win, lane >> 2);
    const bool shave = __shfl_sync(kAll, (int)have, lane >> 2) != 0;
    bool todo = have && lane < kLookRow;
    double d = 0.0;
    if (shave) {
        int k = swin * N - 2 + (lane & 3) * ((R - 1) / 3);
        k = k < 2 ? 2 : k > a.n - 3 ? a.n - 3 : k;  // an interior cell
        d = a.in[LineGeom<1>(a, srow).at(k)];
    }
    double dt;
    if (!sweep_clock(a, dt)) return;
    if (S::steady_params(Cs, dt / P.dx)) {  // warp-uniform
        const double d0 = __shfl_sync(kAll, d, lane & ~3);
        const unsigned agree = __ballot_sync(kAll, shave && same_bits(d, d0));
        for (int i = 0; i < kLookRow; i++) {
            if ((agree >> (4 * i) & 15u) != 15u) continue;  // warp-uniform
            const int c = __shfl_sync(kAll, win, i) * N;
            const LineGeom<1> g(a, __shfl_sync(kAll, row, i));
            // Compared with an output cell (c, but for the row's first window).
            const Cons u0 = load_interior<1>(a, g, c < 2 ? 2 : c);
            bool ok = can_be_steady<S>(u0);
#pragma unroll
            for (int q0 = 0; q0 < Q; q0 += kLookLoads) {
                Cons u[kLookLoads];
#pragma unroll
                for (int j = 0; j < kLookLoads; j++) {
                    const int k = c - 2 + lane + 32 * (q0 + j);
                    u[j] = u0;
                    // Ghost cells are filled on load (and again by the second
                    // launch if the window is not steady).
                    if (k >= 0 && k < a.n) u[j] = load_cell<1>(a, g, k);
                }
#pragma unroll
                for (int j = 0; j < kLookLoads; j++) ok = ok && alike(u[j], u0);
            }
            if (!__all_sync(kAll, ok)) continue;
            if (lane == i) todo = false;
            const Cons o = steady_update(u0);
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const int r = lane + 32 * q, k = c - 2 + r;
                if (r >= 2 && r < 2 + N && k >= 2 && k < a.n - 2) store_cell<1>(a, g, k, o);
            }
            if (a.courant) take_courant<1, S>(Cs, o, cx, cy);
        }
    }
    list_windows(a, todo, row, win);
}

// Along y: a warp looks at one window row of 32 columns (32 / C groups), one
// column a lane.
template <class S, int T, int C>
__device__ __forceinline__ void look_columns(const SweepArgs& a, const Phys& P,
                                             const typename S::Consts& Cs, int warp, double& cx,
                                             double& cy) {
    constexpr int R = T / C, N = R - 4;
    constexpr unsigned kAll = 0xffffffffu, kGroup = (1u << C) - 1u;
    const int lane = threadIdx.x & 31, first = lane / C * C;  // this group's first lane
    const CoopGrid<2, T, C> grid(a);
    const int across = (grid.groups * C + 31) / 32;
    const int row = warp / across, i0 = (warp - row * across) * 32;
    if (row >= grid.nwin) return;  // warp-uniform
    const int win = a.w_lo + row, c = win * N, l = i0 + lane - 2;
    const bool has = l >= 0 && l < a.nlines;
    const LineGeom<2> g(a, l);
    bool steady = false;  // this lane's group
    // Compared with an output cell (c, but for the line's first window).
    const int kref = c < 2 ? 2 : c;
    bool ok = true;
    if (has) {
        const double d0 = a.in[g.at(kref)];
#pragma unroll
        for (int s = 1; s < 4; s++) {
            int k = c - 2 + s * ((R - 1) / 3);
            k = k > a.n - 3 ? a.n - 3 : k;
            ok = same_bits(a.in[g.at(k)], d0) && ok;
        }
    }
    double dt;
    if (!sweep_clock(a, dt)) return;
    if (S::steady_params(Cs, dt / P.dx)) {  // warp-uniform
        steady = (__ballot_sync(kAll, ok) >> first & kGroup) == kGroup;
        if (__any_sync(kAll, steady)) {
            Cons u0{1.0, 0.0, 0.0, 1.0};
            const bool look = has && steady;
            if (look) u0 = load_interior<2>(a, g, kref);
            ok = !look || can_be_steady<S>(u0);
#pragma unroll 1
            for (int r0 = 0; r0 < R; r0 += kLookLoads) {
                Cons u[kLookLoads];
#pragma unroll
                for (int j = 0; j < kLookLoads; j++) {
                    const int k = c - 2 + r0 + j;
                    u[j] = u0;
                    if (look && k >= 0 && k < a.n) u[j] = load_cell<2>(a, g, k);
                }
#pragma unroll
                for (int j = 0; j < kLookLoads; j++) ok = ok && alike(u[j], u0);
            }
            const unsigned same = __ballot_sync(kAll, ok);  // by the whole warp
            steady = steady && (same >> first & kGroup) == kGroup;
            if (has && steady) {
                const Cons o = steady_update(u0);
                const int k0 = c < 2 ? 2 : c, k1 = c + N < a.n - 2 ? c + N : a.n - 2;
                for (int k = k0; k < k1; k++) store_cell<2>(a, g, k, o);
                if (a.courant) take_courant<2, S>(Cs, o, cx, cy);
            }
        }
    }
    // A group exists when any of its columns does.
    const bool exists = (__ballot_sync(kAll, has) >> first & kGroup) != 0u;
    list_windows(a, exists && !steady && lane == first, i0 + first - 2, win);
}

template <class S, int DIR, int T, int C>
__device__ __forceinline__ void steady_body(const SweepArgs& a, const Phys& P) {
    const int warp = (int)(blockIdx.x * (kLookThreads / 32) + (threadIdx.x >> 5));
    const typename S::Consts Cs = S::consts(P);
    double cx = 0.0, cy = 0.0;
    if constexpr (DIR == 1) look_rows<S, T>(a, P, Cs, warp, cx, cy);
    else look_columns<S, T, C>(a, P, Cs, warp, cx, cy);
    if (a.courant) {
        const int slot = cour_slot();
        warp_max_atomic(&a.courant[slot], cx);
        warp_max_atomic(&a.courant[kCourSlots + slot], cy);
    }
}

// The second launch: CTA b of G takes the list's entries b and G + b and then
// claims one after another (the SMs share their issue slots unevenly among
// their CTAs: fixed shares left a quarter of the warp slots idle towards the
// end).  While a window computes, each thread copies its cell of the next one
// into the other half of a shared-memory stage (its own slot only, so the
// copies need no barrier of their own).  The last CTA to finish empties the
// list.
template <class S, int DIR, int T, int C>
__device__ __forceinline__ void coop_list_body(const SweepArgs& a, const Phys& P) {
    __shared__ CoopSmem<S, T> sm;
    __shared__ double stage[2][4][T];
    __shared__ int2 claimed;
    const int t = threadIdx.x;
    const int count = (int)__ldcg(a.todo_count);
    double cx = 0.0, cy = 0.0;
    const int e = blockIdx.x;
    if (e < count) {  // uniform over the CTA
        const typename S::Consts Cs = S::consts(P);
        const double dtdx = (a.clk ? a.clk->dt : a.dt) / P.dx;
        // The entry's window: its first line (group) and number; -1: none.
        auto entry = [&](unsigned i) {
            return i < (unsigned)count ? __ldcg(a.todo + i) : make_int2(0, -1);
        };
        int2 at = entry(e), next = entry(e + gridDim.x);
        int b = 0;
        auto issue = [&](const int2& w, double (*st)[T]) {
            const int l = w.x + t % C;
            coop_stage_issue<DIR, T, C>(a, LineGeom<DIR>(a, l), l >= 0 && l < a.nlines, w.y, st);
        };
        issue(at, stage[0]);
        while (true) {  // ends: each turn takes one of `count` entries
            unsigned claim = 0;
            if (next.y >= 0) {
                issue(next, stage[b ^ 1]);
                if (t == 0) claim = 2 * gridDim.x + atomicAdd(a.todo_count + 2, 1u);
            } else {
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            }
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            const int l = at.x + t % C;
            coop_window<S, DIR, T, C>(a, Cs, l, at.y, dtdx, l >= 0 && l < a.nlines, cx, cy, sm,
                                      stage[b]);
            if (next.y < 0) break;
            if (t == 0) claimed = entry(claim);
            __syncthreads();  // and the window's shared memory is free for the next one
            at = next;
            next = claimed;
            b ^= 1;
        }
        if (a.courant) {
            const int slot = cour_slot();
            warp_max_atomic(&a.courant[slot], cx);
            warp_max_atomic(&a.courant[kCourSlots + slot], cy);
        }
    }
    // Every CTA has read the count and made its claims by its ticket; the last
    // one resets them.
    __syncthreads();
    if (t == 0) {
        __threadfence();
        if (atomicAdd(a.todo_count + 1, 1u) == gridDim.x - 1) {
            a.todo_count[0] = 0u;
            a.todo_count[1] = 0u;
            a.todo_count[2] = 0u;
        }
    }
}

// Threads, lines and outputs per line of the cooperative windows: a row of
// 128 (G = 8: 256) cells along x, 4 columns of 64 (2 of 128) cells along y.
template <int DIR, int G>
struct CoopShape {
    static constexpr int T = DIR == 1 ? 32 * G : 256;
    static constexpr int C = DIR == 1 ? 1 : (G == 4 ? 4 : 2);
    static constexpr int N = T / C - 4;
    static_assert(N == coop_outputs(DIR, G), "window outputs");
    using Grid = CoopGrid<DIR, T, C>;
};

// CTAs of the two launches.
template <int DIR, int T, int C>
inline unsigned steady_ctas(const CoopGrid<DIR, T, C>& grid) {
    const long long warps = DIR == 1
                                ? ((long long)grid.windows() + kLookRow - 1) / kLookRow
                                : (long long)grid.nwin * ((grid.groups * C + 31) / 32);
    return (unsigned)((warps + kLookThreads / 32 - 1) / (kLookThreads / 32));
}
inline unsigned coop_ctas(int windows, int ctas_per_sm) {
    const int wave = device_sm_count() * ctas_per_sm;
    return (unsigned)(windows < wave ? windows : wave);
}
// The two launches of a cooperative sweep over `grid`'s windows.  The first lists
// what the second works and empties; where the second is refused the list is
// emptied here, since its room is that of one sweep's windows and the next
// sweep appends to it.
template <class Grid>
inline cudaError_t launch_coop_pair(void (*look)(SweepArgs, Phys), void (*work)(SweepArgs, Phys),
                                    const Grid& grid, int threads, int threads_per_sm,
                                    const SweepArgs& a, const Phys& P, cudaStream_t s) {
    const int windows = grid.windows();
    if (windows == 0) return cudaSuccess;
    cudaError_t e = launch_sweep_kernel(look, steady_ctas(grid), kLookThreads, s, a, P);
    if (e == cudaSuccess) {
        e = launch_sweep_kernel(work, coop_ctas(windows, threads_per_sm / threads), threads, s, a,
                                P);
        if (e != cudaSuccess) cudaMemsetAsync(a.todo_count, 0, 3 * sizeof(*a.todo_count), s);
    }
    const cudaError_t last = cudaGetLastError();
    return e != cudaSuccess ? e : last;
}

}  // namespace hb
