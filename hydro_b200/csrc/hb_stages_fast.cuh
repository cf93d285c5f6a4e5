// hb_stages_fast.cuh -- the FMA FP64 stage set of the sweep.
//
// The algorithm and the precision of the FP64 restatement (hb_stages.cuh,
// reference citations there), with the arithmetic freed from the reference's
// operation order:
//   * multiply-adds are fused where the code writes fma; the translation unit
//     is built without contraction (--fmad=false), so that a stage rounds the
//     same way in every kernel that calls it;
//   * divisions become multiplications by reciprocals, one reciprocal per
//     denominator, and square roots products with reciprocal square roots;
//     both come from the hardware approximation, refined by two Newton-Raphson
//     steps or one step of fourth order (hb_fastmath.cuh), to within about an
//     ulp.  1/rho and 1/c go from the primitives to the trace, 1/W_K from the iteration to what follows it;
//   * the Newton iteration on p* carries W^2 = c_K + gamma gamma6 rho_K (p - p_K)
//     and 1/W instead of W, and its step is (u*_l - u*_r) / (1/q_l + 1/q_r), the
//     reference's q_l q_r / (q_l + q_r) (u*_l - u*_r) with one reciprocal
//     (riemann.c:136-150).
// Each result differs from the reference's by a few ulps per operation; the
// state stays within 1e-12 (relative, per cell) of the reference's over the
// 200-step 4096^2 centred-blast run (tests/test_gpu_fast.py).  It is not
// bitwise: the Newton stopping test |dp / p| <= 1e-6 may take one iteration
// more or fewer than the reference's where the ratio lies within rounding of
// the threshold, and min/max selections in the limiters may go the other way
// on near-ties.
#pragma once

#include "hb_fastmath.cuh"
#include "hb_stages.cuh"

namespace hb {

// sqrt(x) for x >= 0 as x / sqrt(x) (0 for x = 0; the approximation of
// rsqrt(0) is infinite).
__device__ __forceinline__ double sqrt64(double x) {
    return x > 0.0 ? x * rsqrt64_quartic(x) : 0.0;
}

struct FastConsts {
    Phys P;
    double inv_slope;  // 1 / slope_type
    double gg6;        // gamma gamma6
};

// What the primitives step hands to the trace step: the sound speed c, 1/c and
// 1/rho.
struct SoundD {
    double c, ic, ir;
};

struct FastStages {
    using Consts = FastConsts;
    using Prim = hb::Prim;
    using Flux = Cons;
    using Real = double;   // element type of Prim
    using Sound = SoundD;
    using TraceK = hb::TraceK;
    // Staging the y march's cells by cp.async (the mixed set's column ring)
    // measured slower for the FP64 sets (4096^2: 0.791 against 0.760 ms).
    static constexpr bool async_ring = false;
    static constexpr int ring_ahead = 1;      // rows the ring copies ahead
    static constexpr int cells_per_lane = 1;

    static __device__ __forceinline__ Consts consts(const Phys& P) {
        FastConsts C;
        C.P = P;
        C.inv_slope = 1.0 / P.slope_type;
        C.gg6 = P.gamma * P.gamma6;
        return C;
    }
    static __device__ __forceinline__ Prim zero_prim() { return Prim{0.0, 0.0, 0.0, 0.0}; }
    static __device__ __forceinline__ Flux zero_flux() { return Flux{0.0, 0.0, 0.0, 0.0}; }
    static __device__ __forceinline__ Sound zero_sound() { return Sound{0.0, 0.0, 0.0}; }
    static __device__ __forceinline__ TraceK trace_constants(const Consts& C, double dtdx) {
        return hb::trace_constants(C.P.scheme, dtdx);
    }
    static __device__ __forceinline__ bool second_order(const Consts& C) {
        return C.P.iorder != 1;
    }

    // See steady_update: with |rho| within 2^+-100, momenta and energy below
    // 2^100, velocities stay below 2^200 and the flux below 2^700; the floors
    // and gamma keep pressure and sound speed normal and positive.
    static __device__ __forceinline__ bool steady_params(const Consts& C, double dtdx) {
        return C.P.gamma > 1.0 + 0x1p-20 && C.P.gamma < 256.0 && C.P.smallr > 0x1p-100 &&
               C.P.smallp > 0x1p-200 && C.P.smallp < 1.0 && dtdx > 0.0 && dtdx < 0x1p200;
    }
    static __device__ __forceinline__ bool steady_cell(const Cons& u) {
        return cell_within<-100, 100, 100, 100>(u);
    }

    // constoprim.c:37-52, equation_of_state.c:41-48.
    static __device__ __forceinline__ void prim(const Consts& C, const Cons& u, Prim& q,
                                                Sound& s) {
        const Phys& P = C.P;
        const double r = fmax(u.d, P.smallr);
        const double ir = rcp64(r);
        const double un = u.mn * ir;
        const double ut = u.mt * ir;
        const double e = fma(u.e, ir, -0.5 * fma(un, un, ut * ut));
        const double p = fmax(P.gm1 * r * e, r * P.smallp);
        q = Prim{r, un, ut, p};
        const double c2 = P.gamma * p * ir;
        const double ic = c2 > 0.0 ? rsqrt64_quartic(c2) : 0.0;  // no pressure, no floor: c = 0
        s = Sound{c2 * ic, ic, ir};
    }

    // slope.c:37-50.
    static __device__ __forceinline__ double slope1(const Consts& C, double qm, double q0,
                                                    double qp) {
        double dlft, drgt, dcen;
        if (C.P.unit_slope) {
            dlft = q0 - qm;
            drgt = qp - q0;
            dcen = 0.5 * (dlft + drgt);
        } else {
            dlft = C.P.slope_type * (q0 - qm);
            drgt = C.P.slope_type * (qp - q0);
            dcen = 0.5 * (dlft + drgt) * C.inv_slope;
        }
        const bool llftrgt = (dlft * drgt) <= 0.0;
        const double m = llftrgt ? 0.0 : fmin(fmin(fabs(dlft), fabs(drgt)), fabs(dcen));
        return (dcen > 0.0) ? m : -m;
    }
    static __device__ __forceinline__ void slope4(const Consts& C, const Prim& a, const Prim& b,
                                                  const Prim& c, Prim& dq) {
        if (hb::flat3(a, b, c)) {  // flat: every slope is -0, as slope1 computes
            dq = Prim{-0.0, -0.0, -0.0, -0.0};
            return;
        }
        dq.r = slope1(C, a.r, b.r, c.r);
        dq.u = slope1(C, a.u, b.u, c.u);
        dq.v = slope1(C, a.v, b.v, c.v);
        dq.p = slope1(C, a.p, b.p, c.p);
    }

    // trace.c:63-123, with the factor -1/2 of the characteristic amplitudes
    // folded into them once for both sides.
    static __device__ __forceinline__ void trace(const TraceK& K, const Prim& q, const Prim& dq,
                                                 const Sound& s, Prim& qxm, Prim& qxp) {
        if (dq.r == 0.0 && dq.u == 0.0 && dq.v == 0.0 && dq.p == 0.0) {
            // A flat cell: every characteristic amplitude is zero, so both
            // traced states are the cell's own (the general form can only
            // differ in the sign of a zero velocity).
            qxp = q;
            qxm = q;
            return;
        }
        const double dtdx = K.dtdx, cc = s.c;
        const double csq = cc * cc;
        const double OrOcc = cc * s.ir;
        const double dprcc = dq.p * s.ir * s.ic;
        const double h = -0.25 * (q.r * s.ic);
        const double am0 = (dprcc - dq.u) * h;                     // -alpham / 2
        const double ap0 = (dprcc + dq.u) * h;                     // -alphap / 2
        const double az0 = -0.5 * fma(-dq.p, s.ic * s.ic, dq.r);   // -alpha0r / 2
        const double av0 = -0.5 * dq.v;                            // -alpha0v / 2
        const double upcc = q.u + cc, umcc = q.u - cc;
        // The thresholds are out of reach of a CFL-limited step in MUSCL
        // (hb_stages.cuh, trace1).
        double spm = fma(umcc, dtdx, 1.0), spp = fma(upcc, dtdx, 1.0), spz = fma(q.u, dtdx, 1.0);
        double smm = fma(umcc, dtdx, -1.0), smp = fma(upcc, dtdx, -1.0);
        double smz = fma(q.u, dtdx, -1.0);
        if (!(fabs(q.u) + cc < K.zeror)) {
            if (umcc >= K.zeror) spm = K.project;
            if (upcc >= K.zeror) spp = K.project;
            if (q.u >= K.zeror) spz = K.project;
            if (umcc <= K.zerol) smm = -K.project;
            if (upcc <= K.zerol) smp = -K.project;
            if (q.u <= K.zerol) smz = -K.project;
        }
        double ap = spp * ap0, am = spm * am0;
        qxp = Prim{q.r + fma(spz, az0, ap + am), fma(ap - am, OrOcc, q.u), fma(spz, av0, q.v),
                   fma(ap + am, csq, q.p)};
        ap = smp * ap0;
        am = smm * am0;
        qxm = Prim{q.r + fma(smz, az0, ap + am), fma(ap - am, OrOcc, q.u), fma(smz, av0, q.v),
                   fma(ap + am, csq, q.p)};
    }

    // riemann.c:89-258 and cmpflx.c:52-73, with the C99 selection order.
    static __device__ __forceinline__ Flux riemann(const Consts& C, const Prim& ql,
                                                   const Prim& qr) {
        const Phys& P = C.P;
        const double rl = fmax(ql.r, P.smallr), ul = ql.u;
        const double pl = fmax(ql.p, rl * P.smallp);
        const double rr = fmax(qr.r, P.smallr), ur = qr.u;
        const double pr = fmax(qr.p, rr * P.smallp);
        double gr, gu, gp, gv;  // the state sampled at the interface
        if (pl == pr && ul == ur) {
            // Equal pressure and velocity on both sides (at rest, a uniform
            // flow or a pure contact): the exact solution p* = p, u* = u, where
            // the reference's iteration lands within rounding of p; the
            // interface samples the upwind side's state (the right for u = 0).
            const bool left = ul > 0.0;
            gr = left ? rl : rr;
            gu = ul;
            gp = pl;
            gv = left ? ql.v : qr.v;
        } else {
            const double cl = P.gamma * pl * rl;
            const double cr = P.gamma * pr * rr;
            // W_K^2 = c_K (1 + gamma6 (p - p_K) / p_K) = c_K + k_K (p - p_K).
            const double kl = C.gg6 * rl, kr = C.gg6 * rr;
            double il = rsqrt64_quartic(cl), ir = rsqrt64_quartic(cr);  // 1 / W
            const double wl0 = cl * il, wr0 = cr * ir;
            double pst = fmax(
                fma(wl0 * wr0, ul - ur, fma(wr0, pl, wl0 * pr)) * rcp64(wl0 + wr0), 0.0);
            for (int iter = 0; iter < P.niter; iter++) {
                const double wl2 = fma(kl, pst - pl, cl);
                const double wr2 = fma(kr, pst - pr, cr);
                il = rsqrt64_quartic(wl2);
                ir = rsqrt64_quartic(wr2);
                const double dus = fma(-(pst - pl), il, ul) - fma(pst - pr, ir, ur);
                // 2 / q_K = (W^2 + c_K) / W^3
                const double iql = (wl2 + cl) * (il * il * il);
                const double iqr = (wr2 + cr) * (ir * ir * ir);
                double delp = 2.0 * dus * rcp64(iql + iqr);
                delp = delp > -pst ? delp : -pst;
                pst += delp;
                if (!(fabs(delp) > 1e-6 * (pst + P.smallpp))) break;
            }
            const double pstar = pst;

            const double wl2 = fma(kl, pstar - pl, cl);
            const double wr2 = fma(kr, pstar - pr, cr);
            il = rsqrt64_quartic(wl2);
            ir = rsqrt64_quartic(wr2);
            // Grouped so that a mirror pair (a reflecting wall) gives 0 exactly.
            const double ustar = 0.5 * ((ul + ur) + ((pl - pstar) * il - (pr - pstar) * ir));
            const bool left = ustar > 0.0;
            const double ro = left ? rl : rr;
            const double uo = left ? ul : ur;
            const double po = left ? pl : pr;
            const double iwo = left ? il : ir;
            const double wo = (left ? wl2 : wr2) * iwo;
            // The selection by comparison, as in the bit-exact set
            // (riemann_flux): the squares decide where they are 1e-9 apart.
            const double su = left ? uo : -uo;
            const bool shock = pstar >= po;
            const double lhs = shock ? wo : P.gamma * po;
            const double rhs = (shock ? su : su * su) * ro;
            gr = ro;
            gu = uo;
            gp = po;
            if (!(lhs < rhs * (1.0 - 1e-9) && (shock || su > P.smallc))) {
                double rstar = ro * rcp64(fma(ro * (po - pstar), iwo * iwo, 1.0));
                rstar = fmax(rstar, P.smallr);
                if ((lhs > rhs * (1.0 + 1e-9) || (!shock && su <= 0.0)) &&
                    (shock || P.gamma * pstar > ustar * ustar * rstar * (1.0 + 1e-9))) {
                    gr = rstar;
                    gu = ustar;
                    gp = pstar;
                } else {
                    const double iro = rcp64(ro);
                    double spout, spin;
                    if (shock) {
                        spin = spout = fma(wo, iro, -su);
                    } else {
                        spout = fmax(P.smallc, sqrt64(fabs(P.gamma * po * iro))) - su;
                        spin = fmax(P.smallc, sqrt64(fabs(P.gamma * pstar * rcp64(rstar)))) -
                               fabs(ustar);
                    }
                    const double scr = fmax(spout - spin, P.smallc + fabs(spout + spin));
                    const double frac =
                        fmax(0.0, fmin(1.0, fma((spout + spin) * rcp64(scr), 0.5, 0.5)));
                    if (!(spout < 0.0)) {
                        const bool star = spin > 0.0;
                        gr = star ? rstar : fma(frac, rstar, (1.0 - frac) * ro);
                        gu = star ? ustar : fma(frac, ustar, (1.0 - frac) * uo);
                        gp = star ? pstar : fma(frac, pstar, (1.0 - frac) * po);
                    }
                }
            }
            gv = left ? ql.v : qr.v;
        }
        Cons f;
        const double mass = gr * gu;
        f.d = mass;
        f.mn = fma(mass, gu, gp);
        f.mt = mass * gv;
        const double etot = fma(gp, P.entho, 0.5 * gr * fma(gu, gu, gv * gv));
        f.e = gu * (etot + gp);
        return f;
    }

    // conservar.c:166-172.
    static __device__ __forceinline__ Cons update(const Cons& u, const Flux& fl, const Flux& fr,
                                                  double dtdx) {
        return Cons{fma(fl.d - fr.d, dtdx, u.d), fma(fl.mn - fr.mn, dtdx, u.mn),
                    fma(fl.mt - fr.mt, dtdx, u.mt), fma(fl.e - fr.e, dtdx, u.e)};
    }

    // ComputeQEforRow.c:31-47, equation_of_state.c:41-48, courantOnXY.c:44-45.
    static __device__ __forceinline__ void courant(const Consts& C, const Cons& u, double& cn,
                                                   double& ct) {
        Prim q;
        Sound s;
        prim(C, u, q, s);
        cn = s.c + fabs(q.u);
        ct = s.c + fabs(q.v);
    }
};

}  // namespace hb
