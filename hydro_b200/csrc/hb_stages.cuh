// hb_stages.cuh -- per-cell / per-interface device functions of the HydroC
// Godunov/MUSCL step, FP64.
//
// Every function restates the arithmetic of the reference
// (HydroC/HydroC99_2Domp/Src, cited per function) with the same IEEE
// operations in the same order.  The translation unit that includes this file
// is compiled with --fmad=false and IEEE division / square root, so each
// operation is rounded once, exactly as in the reference's C build (gcc -O3
// -mavx2, no FMA): the kernels reproduce the reference bit for bit.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace hb {

// Primitive variables of one cell in line orientation: density, velocity
// normal to the sweep, transverse velocity, pressure.
struct Prim {
    double r, u, v, p;
};

// Conservative variables in line orientation: rho, normal momentum,
// transverse momentum, total energy.
struct Cons {
    double d, mn, mt, e;
};

// 2^DLO <= rho < 2^DHI, |momenta| < 2^MHI and |E| < 2^EHI (exponent fields).
template <int DLO, int DHI, int MHI, int EHI>
__device__ __forceinline__ bool cell_within(const Cons& u) {
    constexpr int M = 0x7fffffff;
    return (unsigned)(__double2hiint(u.d) - ((1023 + DLO) << 20)) < (unsigned)((DHI - DLO) << 20) &&
           (__double2hiint(u.mn) & M) < ((1023 + MHI) << 20) &&
           (__double2hiint(u.mt) & M) < ((1023 + MHI) << 20) &&
           (__double2hiint(u.e) & M) < ((1023 + EHI) << 20);
}

// Constants of one run, derived on the host with the reference's formulas.
struct Phys {
    double gamma, gm1;    // gamma, gamma - 1 (equation_of_state.c:42)
    double smallr, smallc;
    double smallp;        // smallc^2 / gamma (equation_of_state.c:25, riemann.c:34)
    double gamma6;        // (gamma + 1) / (2 gamma) (riemann.c:35)
    double smallpp;       // smallr * smallp (riemann.c:36)
    double entho;         // 1 / (gamma - 1) (cmpflx.c:27)
    double slope_type;
    double dx;
    int niter;            // niter_riemann
    int iorder;           // 1: first order (dq = 0)
    int scheme;           // 1 muscl, 2 plmde, 3 collela
    int unit_slope;       // slope_type == 1.0 (x*1 and x/1 are exact: skipped)
};

// utils.h:9-11 MAX(x, y): x > y ? x : y.
__device__ __forceinline__ double omax(double x, double y) { return x > y ? x : y; }

// C99 fmax / fmin as glibc evaluates them for non-NaN operands: x when
// x >= y (resp. x <= y), so a tie between +0 and -0 returns the first operand,
// which PTX max.f64/min.f64 do not promise.  (NaN operands, which a valid
// state never produces, are not given C99's "return the other operand" rule.)
__device__ __forceinline__ double cfmax(double x, double y) { return x >= y ? x : y; }
__device__ __forceinline__ double cfmin(double x, double y) { return x <= y ? x : y; }

// a / b, IEEE-rounded, for a denominator b that is finite and nonzero (every
// call site divides by a positive quantity of a valid state).  A zero
// numerator gives its signed zero as the product a * b, which has the
// quotient's sign and value, without entering the division: the IEEE division
// sequence sends a zero numerator down its slow path (a called subroutine),
// and the limiter zeroes slopes at every extremum.  Nonzero numerators take
// the ordinary division, so the result is bitwise a / b in every case.
__device__ __forceinline__ double zdiv(double a, double b) {
    if (a == 0.0) return a * b;
    return a / b;
}

// Quotients that share a denominator b > 0.  y is 1 / b correctly rounded and
// y + yl is 1 / b to about twice FP64: one reciprocal serves every numerator,
// at 4 operations each.  The method is Markstein's (IBM J. Res. Dev. 34, 1990;
// Muller et al., Handbook of Floating-Point Arithmetic, section 4.7):
//  - a reciprocal within 1 ulp, corrected once by its exact FMA residual, is
//    correctly rounded unless b's significand is all ones;
//  - q within 1 ulp of a / b has an exact residual a - b q, and q corrected by
//    it with the rounded reciprocal is a / b correctly rounded.
// Here q = a y + a yl is within 0.5 ulp and a rounding of its small term.  Both
// facts need every quantity in the normal range, which range_bits tests, and
// low words of ones are left to the division.
struct Recip {
    double b, y, yl;
};

// Nonzero in mask 0x60000000 unless 2^-255 <= |x| < 2^257 (the exponent field
// lies in [768, 1280)).
__device__ __forceinline__ int range_bits(double x) { return __double2hiint(x) - 0x30000000; }
constexpr int kRangeMask = 0x60000000;
// The same for 2^-128 <= |x| < 2^128 with mask 0x70000000.
__device__ __forceinline__ int range_bits128(double x) { return __double2hiint(x) - 0x37f00000; }
constexpr int kRangeMask128 = 0x70000000;

// 1 / b correctly rounded (see Recip): the hardware approximation, one cubic
// step (relative error e -> e^3, below 1 ulp), one Markstein correction.
__device__ __forceinline__ double recip_rn(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = fma(-b, y, 1.0);
    e = fma(e, e, e);
    y = fma(y, e, y);
    e = fma(-b, y, 1.0);
    return fma(y, e, y);
}

__device__ __forceinline__ Recip make_recip(double b) {
    const double y = recip_rn(b);
    return Recip{b, y, fma(-b, y, 1.0) * y};
}

__device__ __forceinline__ double quot(double a, const Recip& R) {
    const double q = fma(a, R.y, a * R.yl);
    return fma(fma(-R.b, q, a), R.y, q);
}

// The same without yl (one operation more, two registers less): the first
// correction brings a y within 1 ulp, the second rounds correctly.
__device__ __forceinline__ double quot1(double a, double b, double y) {
    double q = a * y;
    q = fma(fma(-b, q, a), y, q);
    return fma(fma(-b, q, a), y, q);
}

__device__ __forceinline__ bool is_zero(double x) {
    return ((__double2hiint(x) << 1) | __double2loint(x)) == 0;
}

// constoprim.c:37-52 then equation_of_state.c:41-48, the four divisions by rho
// as quotients of one reciprocal (by zdiv out of their range).
__device__ __forceinline__ void cons_to_prim(const Phys& P, const Cons& u, Prim& q, double& c) {
    const double r = omax(u.d, P.smallr);
    const Recip R = make_recip(r);
    // A zero momentum's quotient is the zero itself (rho > 0).
    const bool zn = is_zero(u.mn), zt = is_zero(u.mt);
    double un = quot(u.mn, R), ut = quot(u.mt, R);
    const double ue = quot(u.e, R);
    int bad = range_bits(r) | range_bits(u.e) | range_bits(ue);
    bad |= zn ? 0 : (range_bits(u.mn) | range_bits(un));
    bad |= zt ? 0 : (range_bits(u.mt) | range_bits(ut));
    un = zn ? u.mn : un;
    ut = zt ? u.mt : ut;
    const double eken = 0.5 * ((un * un) + (ut * ut));
    const double e = ue - eken;
    double base = P.gm1 * r * e;
    base = omax(base, r * P.smallp);
    const double gb = P.gamma * base;
    const double c2 = quot(gb, R);
    bad |= range_bits(gb) | range_bits(c2);
    q = Prim{r, un, ut, base};
    double cc = c2;
    if ((bad & kRangeMask) != 0 || __double2loint(r) == -1) {
        q.u = zdiv(u.mn, r);
        q.v = zdiv(u.mt, r);
        const double ek = 0.5 * ((q.u * q.u) + (q.v * q.v));
        q.p = omax(P.gm1 * r * (u.e / r - ek), r * P.smallp);
        cc = P.gamma * q.p / r;
    }
    c = sqrt(cc);
}

// slope.c:37-50 for one variable.
template <bool UNIT>
__device__ __forceinline__ double slope1(double st, double qm, double q0, double qp) {
    double dlft, drgt, dcen;
    if (UNIT) {
        dlft = q0 - qm;
        drgt = qp - q0;
        dcen = 0.5 * (dlft + drgt);
    } else {
        dlft = st * (q0 - qm);
        drgt = st * (qp - q0);
        dcen = 0.5 * (dlft + drgt) / st;
    }
    // dsgn * fmin((1 - llftrgt) * t1, |dcen|) of the reference, written as a
    // select: for finite slopes (1 - llftrgt) * t1 is t1 or +0, fmin(+0, x >= 0)
    // is +0, and (-1) * m is -m exactly, so the bits are the same.
    const bool llftrgt = (dlft * drgt) <= 0.0;
    const double t1 = cfmin(fabs(dlft), fabs(drgt));
    const double m = llftrgt ? 0.0 : cfmin(t1, fabs(dcen));
    return (dcen > 0.0) ? m : -m;
}

// A flat neighbourhood (every variable's two differences exactly zero, which
// also excludes infinities) gives -0 for every slope: +0 differences, +0
// centred slope, a limited magnitude of +0 and the negative branch of the
// sign select, the same bits slope1 computes.
__device__ __forceinline__ bool flat3(const Prim& a, const Prim& b, const Prim& c) {
    return b.r - a.r == 0.0 && c.r - b.r == 0.0 && b.u - a.u == 0.0 && c.u - b.u == 0.0 &&
           b.v - a.v == 0.0 && c.v - b.v == 0.0 && b.p - a.p == 0.0 && c.p - b.p == 0.0;
}

template <bool UNIT>
__device__ __forceinline__ void slope4(double st, const Prim& a, const Prim& b, const Prim& c,
                                       Prim& dq) {
    if (flat3(a, b, c)) {
        dq = Prim{-0.0, -0.0, -0.0, -0.0};
        return;
    }
    dq.r = slope1<UNIT>(st, a.r, b.r, c.r);
    dq.u = slope1<UNIT>(st, a.u, b.u, c.u);
    dq.v = slope1<UNIT>(st, a.v, b.v, c.v);
    dq.p = slope1<UNIT>(st, a.p, b.p, c.p);
}

// Scheme constants of trace.c:30-46.
struct TraceK {
    double dtdx, zerol, zeror, project;
};

__device__ __forceinline__ TraceK trace_constants(int scheme, double dtdx) {
    TraceK k;
    k.dtdx = dtdx;
    k.zerol = 0.0;
    k.zeror = 0.0;
    k.project = 0.0;
    if (scheme == 1) {
        k.zerol = -100.0 / dtdx;
        k.zeror = 100.0 / dtdx;
        k.project = 1.0;
    }
    if (scheme == 2) {
        k.project = 1.0;
    }
    return k;
}

// trace.c:63-123 for one cell: left (qxm) and right (qxp) states.
__device__ __forceinline__ void trace1(const TraceK& K, const Prim& q, const Prim& dq, double cc,
                                       Prim& qxm, Prim& qxp) {
    const double dtdx = K.dtdx;
    // With every slope zero (of either sign), the four factors below only scale
    // signed zeros, and any positive finite factor gives those zeros the same
    // signs: such a cell (the flat cells of a state at rest, or extrema) takes 1
    // for each and skips both IEEE divisions, with the same bits.  The range
    // test keeps the general factors finite and nonzero where this is taken.
    const bool zero_slopes = dq.r == 0.0 && dq.u == 0.0 && dq.v == 0.0 && dq.p == 0.0 &&
                             cc > 1e-100 && cc < 1e100 && q.r > 1e-100 && q.r < 1e100;
    double csq = 1.0, rOcc = 1.0, OrOcc = 1.0, rcc = 1.0;
    if (!zero_slopes) {
        csq = cc * cc;
        rOcc = q.r / cc;
        OrOcc = cc / q.r;
        rcc = q.r * cc;
    }
    double dprcc = zdiv(dq.p, rcc);
    double alpham = 0.5 * (dprcc - dq.u) * rOcc;
    double alphap = 0.5 * (dprcc + dq.u) * rOcc;
    double alpha0r = dq.r - zdiv(dq.p, csq);
    double alpha0v = dq.v;
    double upcc = q.u + cc;
    double umcc = q.u - cc;
    double upccx = upcc * dtdx;
    double umccx = umcc * dtdx;
    double ux = q.u * dtdx;

    // MUSCL's thresholds are +-100 dx/dt, which no wave of a CFL-limited step
    // reaches: |u| + c below them decides all six selections at once.
    double spminus = umccx + 1.0, spplus = upccx + 1.0, spzero = ux + 1.0;
    double smminus = umccx - 1.0, smplus = upccx - 1.0, smzero = ux - 1.0;
    if (!(fabs(q.u) + cc < K.zeror)) {
        if (umcc >= K.zeror) spminus = K.project;
        if (upcc >= K.zeror) spplus = K.project;
        if (q.u >= K.zeror) spzero = K.project;
        if (umcc <= K.zerol) smminus = -K.project;
        if (upcc <= K.zerol) smplus = -K.project;
        if (q.u <= K.zerol) smzero = -K.project;
    }
    double ap = -0.5 * spplus * alphap;
    double am = -0.5 * spminus * alpham;
    double azr = -0.5 * spzero * alpha0r;
    double azv = -0.5 * spzero * alpha0v;
    qxp.r = q.r + (ap + am + azr);
    qxp.u = q.u + (ap - am) * OrOcc;
    qxp.v = q.v + (azv);
    qxp.p = q.p + (ap + am) * csq;

    ap = -0.5 * smplus * alphap;
    am = -0.5 * smminus * alpham;
    azr = -0.5 * smzero * alpha0r;
    azv = -0.5 * smzero * alpha0v;
    qxm.r = q.r + (ap + am + azr);
    qxm.u = q.u + (ap - am) * OrOcc;
    qxm.v = q.v + (azv);
    qxm.p = q.p + (ap + am) * csq;
}

// cmpflx.c:52-73.
__device__ __forceinline__ Cons state_flux(const Phys& P, double gr, double gu, double gv,
                                           double gp) {
    Cons f;
    const double mass = gr * gu;
    f.d = mass;
    f.mn = mass * gu + gp;
    f.mt = mass * gv;
    const double ekin = 0.5 * gr * ((gu * gu) + (gv * gv));
    const double etot = gp * P.entho + ekin;
    f.e = gu * (etot + gp);
    return f;
}

// a / b with y = 1 / b from recip_rn, or by the division.
__device__ __forceinline__ double quot_or_div(double a, double b, double y, bool fast) {
    if (fast) return quot1(a, b, y);
    return zdiv(a, b);
}

// riemann.c:89-110 (first guess), :126-156 (Newton iterations on p*, at most
// niter, stopping per interface once |dp/p| <= 1e-6), :175-258 (sampling, with
// the C99 selection order: outer state if spout < 0, else star state if
// spin > 0, else the blend), then the flux of the Godunov state
// (cmpflx.c:52-73).  ql = qxm of the cell left of the interface, qr = qxp of
// the cell to its right (qleftright.c:45-46).
//
// Every number that reaches the flux carries the reference's bits; what is
// only compared is compared without being formed:
//  - the Newton step dp = q_l q_r / (q_l + q_r) du goes into p* + dp and into
//    the stop test.  With one reciprocal and no rounding order to keep it is
//    within 2^-49 (relative) of the reference's three divisions: 7 roundings
//    there and 7 here, 2^-53 each.  p* + dp (1 +- 2^-49) rounding to one number
//    is therefore the reference's, and so is a stop test that holds with 1e-9
//    to spare; otherwise the step is formed by its divisions (dp is mostly
//    1e-3 to 1e-8 of p*: rarely).
//  - the selection asks only for the signs of spout and spin, which compare
//    W/rho, c and c* with a velocity: their squares do, without the division
//    and the square root, unless they lie within 1e-9 of each other or the
//    state is a blend.
__device__ __forceinline__ Cons riemann_flux(const Phys& P, const Prim& ql, const Prim& qr) {
    const double gamma = P.gamma, smallr = P.smallr, smallp = P.smallp;
    const double gamma6 = P.gamma6;
    constexpr double kUp = 1.0 + 1e-9, kDown = 1.0 - 1e-9;

    const double rl = cfmax(ql.r, smallr);
    const double ul = ql.u;
    const double pl = cfmax(ql.p, rl * smallp);
    const double rr = cfmax(qr.r, smallr);
    const double ur = qr.u;
    const double pr = cfmax(qr.p, rr * smallp);
    // Densities and pressures within 2^+-128 and gamma within 2^+-8 keep every
    // product below normal; low words of ones have no rounded reciprocal here
    // (Recip).
    const bool fast =
        ((range_bits128(rl) | range_bits128(rr) | range_bits128(pl) | range_bits128(pr)) &
         kRangeMask128) == 0 &&
        (unsigned)(__double2hiint(gamma) - 0x3f700000) < 0x01000000u &&
        __double2loint(pl) != -1 && __double2loint(pr) != -1;
    const double cl = gamma * pl * rl;
    const double cr = gamma * pr * rr;
    double wl = sqrt(cl);
    double wr = sqrt(cr);
    double pstar = cfmax(((wr * pl + wl * pr) + wl * wr * (ul - ur)) / (wl + wr), 0.0);
    const double yl = recip_rn(pl), yr = recip_rn(pr);

    for (int iter = 0; iter < P.niter; iter++) {
        const double pst = pstar;
        const double wwl = sqrt(cl * (1.0 + quot_or_div(gamma6 * (pst - pl), pl, yl, fast)));
        const double wwr = sqrt(cr * (1.0 + quot_or_div(gamma6 * (pst - pr), pr, yr, fast)));
        const double usl = ul - zdiv(pst - pl, wwl);
        const double usr = ur + zdiv(pst - pr, wwr);
        const double dus = usl - usr;
        const double sl = wwl * wwl, sr = wwr * wwr;
        const double nl = 2.0 * wwl * sl, nr = 2.0 * wwr * sr;  // q_K = n_K / d_K
        const double dl = sl + cl, dr = sr + cr;
        const double den = fma(nr, dl, nl * dr);
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(den));
        double e = fma(-den, y, 1.0);
        e = fma(e, e, e);
        y = fma(y, e, y);
        double delp = dus * (nr * nl) * y;
        pstar = fma(delp, 1.0 + 0x1p-49, pst);
        const bool same = pstar == fma(delp, 1.0 - 0x1p-49, pst) && pstar > 0x1p-300;
        const double lim = 1e-6 * (pstar + P.smallpp);
        bool go = fabs(delp) > lim * kUp;
        if (!(same && fast && (go || fabs(delp) < lim * kDown))) {
            const double qlw = nl / dl, qrw = nr / dr;
            delp = omax(qrw * qlw / (qrw + qlw) * dus, -pst);
            pstar = pst + delp;
            go = fabs(zdiv(delp, pstar + P.smallpp)) > 1e-6;
        }
        if (!go) break;
    }

    wr = sqrt(cr * (1.0 + quot_or_div(gamma6 * (pstar - pr), pr, yr, fast)));
    wl = sqrt(cl * (1.0 + quot_or_div(gamma6 * (pstar - pl), pl, yl, fast)));
    const double ustar = 0.5 * (ul + zdiv(pl - pstar, wl) + ur - zdiv(pr - pstar, wr));
    const bool left = ustar > 0.0;
    const double ro = left ? rl : rr;
    const double uo = left ? ul : ur;
    const double po = left ? pl : pr;
    const double wo = left ? wl : wr;

    const double su = left ? uo : -uo;
    const bool shock = pstar >= po;
    // Shock: spout = spin = W/rho - su.  Rarefaction: spout = max(smallc, c) - su.
    const double lhs = shock ? wo : gamma * po;
    const double rhs = (shock ? su : su * su) * ro;
    double gr = ro, gu = uo, gp = po;
    if (!(lhs < rhs * kDown && (shock || su > P.smallc) && fast)) {
        double rstar = ro / (1.0 + zdiv(ro * (po - pstar), wo * wo));
        rstar = cfmax(rstar, smallr);
        // Rarefaction: spin = max(smallc, c*) - |u*|.
        if ((lhs > rhs * kUp || (!shock && su <= 0.0)) && fast &&
            (shock || gamma * pstar > ustar * ustar * rstar * kUp)) {
            gr = rstar;
            gu = ustar;
            gp = pstar;
        } else {
            double spout, spin;
            if (shock) {
                spout = spin = wo / ro - su;
            } else {
                spout = cfmax(P.smallc, sqrt(fabs(gamma * po / ro))) - su;
                spin = cfmax(P.smallc, sqrt(fabs(gamma * pstar / rstar))) - fabs(ustar);
            }
            const double scr = cfmax(spout - spin, P.smallc + fabs(spout + spin));
            double frac = (1.0 + (spout + spin) / scr) * 0.5;
            frac = cfmax(0.0, cfmin(1.0, frac));
            if (!(spout < 0.0)) {
                const bool star = spin > 0.0;
                gr = star ? rstar : (frac * rstar + (1.0 - frac) * ro);
                gu = star ? ustar : (frac * ustar + (1.0 - frac) * uo);
                gp = star ? pstar : (frac * pstar + (1.0 - frac) * po);
            }
        }
    }
    return state_flux(P, gr, gu, left ? ql.v : qr.v, gp);
}

// conservar.c:166-172: u + (F_left - F_right) * dtdx, difference first.
__device__ __forceinline__ Cons update(const Cons& u, const Cons& fl, const Cons& fr, double dtdx) {
    Cons o;
    o.d = u.d + (fl.d - fr.d) * dtdx;
    o.mn = u.mn + (fl.mn - fr.mn) * dtdx;
    o.mt = u.mt + (fl.mt - fr.mt) * dtdx;
    o.e = u.e + (fl.e - fr.e) * dtdx;
    return o;
}

// Courant speeds of one updated cell: ComputeQEforRow.c:31-47,
// equation_of_state.c:41-48, courantOnXY.c:44-45.  cn / ct: c + |u| along the
// sweep's normal / transverse direction.
__device__ __forceinline__ void courant_speeds(const Phys& P, const Cons& u, double& cn,
                                               double& ct) {
    Prim q;
    double c;
    cons_to_prim(P, u, q, c);
    cn = c + fabs(q.u);
    ct = c + fabs(q.v);
}

// The exact FP64 stage set used by the plain sweep (hb_march.cuh).
template <bool UNIT>
struct ExactStages {
    using Consts = Phys;
    using Prim = hb::Prim;
    using Flux = Cons;
    using Real = double;   // element type of Prim
    using Sound = double;  // the sound speed, from prim to trace
    using TraceK = hb::TraceK;
    // Staging the y march's cells by cp.async (the mixed set's column ring)
    // measured slower for the FP64 sets (4096^2: 0.791 against 0.760 ms).
    static constexpr bool async_ring = false;
    static constexpr int ring_ahead = 1;      // rows the ring copies ahead
    static constexpr int cells_per_lane = 1;  // x sweep window (hb_march.cuh)
    static __device__ __forceinline__ Consts consts(const Phys& P) { return P; }
    static __device__ __forceinline__ Prim zero_prim() { return Prim{0.0, 0.0, 0.0, 0.0}; }
    static __device__ __forceinline__ Flux zero_flux() { return Flux{0.0, 0.0, 0.0, 0.0}; }
    static __device__ __forceinline__ Sound zero_sound() { return 0.0; }
    static __device__ __forceinline__ TraceK trace_constants(const Phys& P, double dtdx) {
        return hb::trace_constants(P.scheme, dtdx);
    }
    static __device__ __forceinline__ bool second_order(const Phys& P) { return P.iorder != 1; }
    // See steady_update: with |rho| within 2^+-100, momenta and energy below
    // 2^100, velocities stay below 2^200 and the flux below 2^700; the floors
    // and gamma keep pressure and sound speed normal and positive.
    static __device__ __forceinline__ bool steady_params(const Consts& P, double dtdx) {
        return P.gamma > 1.0 + 0x1p-20 && P.gamma < 256.0 && P.smallr > 0x1p-100 &&
               P.smallp > 0x1p-200 && P.smallp < 1.0 && dtdx > 0.0 && dtdx < 0x1p200;
    }
    static __device__ __forceinline__ bool steady_cell(const Cons& u) {
        return cell_within<-100, 100, 100, 100>(u);
    }
    static __device__ __forceinline__ void prim(const Phys& P, const Cons& u, Prim& q, double& c) {
        cons_to_prim(P, u, q, c);
    }
    static __device__ __forceinline__ void slope4(const Phys& P, const Prim& a, const Prim& b,
                                                  const Prim& c, Prim& dq) {
        hb::slope4<UNIT>(P.slope_type, a, b, c, dq);
    }
    static __device__ __forceinline__ void trace(const TraceK& K, const Prim& q, const Prim& dq,
                                                 double c, Prim& xm, Prim& xp) {
        trace1(K, q, dq, c, xm, xp);
    }
    static __device__ __forceinline__ Flux riemann(const Phys& P, const Prim& l, const Prim& r) {
        return riemann_flux(P, l, r);
    }
    static __device__ __forceinline__ Cons update(const Cons& u, const Flux& fl, const Flux& fr,
                                                  double dtdx) {
        return hb::update(u, fl, fr, dtdx);
    }
    static __device__ __forceinline__ void courant(const Phys& P, const Cons& u, double& cn,
                                                   double& ct) {
        courant_speeds(P, u, cn, ct);
    }
};

}  // namespace hb
