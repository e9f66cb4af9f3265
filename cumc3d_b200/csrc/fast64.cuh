// fast64.cuh -- the FP64 reconstruction and Riemann arithmetic without
// branches in its divisions and square roots.
//
// The plain forms (mhd_device.cuh) divide with the IEEE operator, one guarded
// division after the other, and the kernels waited out one dependency chain
// after the other (128^3 blast, HLLD: FP64 pipe 45% busy, 51% of issue slots,
// 4 warps per scheduler, 180 us a sweep; this form 63-68%, 101-109 us; WENO-Z
// reconstruction 274 and 190 us).  Here a quotient is a reciprocal refined from the hardware seed
// and one residual correction, straight-line code that the compiler
// interleaves freely; one reciprocal serves every quotient over the same
// divisor; and the operands' exponents are tested on the integer pipe, beside
// the arithmetic, into one flag per cell or face.  Where the flag fails (a
// value outside the tested range, not finite, or a divisor with an all-ones
// mantissa) the caller recomputes the cell with the plain form.
//
// Method: reciprocal by one third-order step, y = y0 (1 + e + e^2) with
// e = 1 - b y0; quotient q = x y, then q + (x - b q) y with the residual from
// one fused multiply-add (Markstein, IBM J. Res. Dev. 34, 1990); square root
// by one third-order step on x^(-1/2) and the same kind of residual
// correction.  The seed is good to 2^-19.9, so y is within 0.51 ulp of 1/b.
// Measured against x / y and sqrt(x) (cumc_check_fast64): no difference in 2^30
// generated pairs or arguments of the ranges used here.  On
// pairs built so that the quotient lies within 2^-52 ulp of a rounding
// boundary (7 of 2^28) the quotient can fall on the other side when the
// divisor's mantissa is above 1.99 (none below); the chance for an arbitrary pair
// is below 2^-70.  Power-of-two numerators over an all-ones divisor, the one case that
// occurs in practice (1 / 0.999...), are excluded by the tests.
#pragma once
#include "mhd_device.cuh"

namespace cumc {

// hardware seeds (PTX rcp.approx.ftz.f64, rsqrt.approx.ftz.f64)
__device__ __forceinline__ double seed_rcp(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    return r;
}
__device__ __forceinline__ double seed_rsqrt(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
// 1/b, not quite correctly rounded (0.51 ulp): the multiplier of quo()
__device__ __forceinline__ double inv64(double b) {
    const double y = seed_rcp(b);
    const double e = __fma_rn(-b, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}
// x / b from y = inv64(b).  POS: b > 0, else b < 0: the residual's sign is
// chosen so that a zero numerator keeps the quotient's sign of zero.
template <bool POS = true>
__device__ __forceinline__ double quo(double x, double b, double y) {
    const double q = __dmul_rn(x, y);
    if (POS) return __fma_rn(-__fma_rn(b, q, -x), y, q);
    return __fma_rn(__fma_rn(-b, q, x), y, q);
}
__device__ __forceinline__ double sqrt64(double x) {
    const double y = seed_rsqrt(x);
    // y / 2 on the integer pipe (the seed is a normal number for a tested x)
    const double h = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
    const double g = __dmul_rn(x, y);
    const double r = __fma_rn(-g, h, 0.5);
    const double c = __dmul_rn(r, __fma_rn(1.5, r, 1.0));
    const double g1 = __fma_rn(g, c, g);
    return __fma_rn(__fma_rn(-g1, g1, x), __fma_rn(h, c, h), g1);
}

// x / 3 for an x whose product with 2^-55 does not underflow: x RN(1/3) plus
// the rounded x (1/3 - RN(1/3)), the sum with one FMA.  Within 2^-52 ulp of
// x / 3 before its rounding, and x / 3 is never nearer than 1/6 ulp to a
// midpoint, so this is the IEEE quotient in two operations (div3: three, any x).
__device__ __forceinline__ double third64(double x) {
    return __fma_rn(x, 1.0 / 3.0, __dmul_rn(x, 0x1p-54 / 3.0));
}

// the high word of 2^e
__device__ __forceinline__ constexpr unsigned hi2(int e) { return (unsigned)(1023 + e) << 20; }
__device__ __forceinline__ unsigned habs(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }
__device__ __forceinline__ unsigned hi64(double x) { return (unsigned)__double2hiint(x); }
__device__ __forceinline__ unsigned lo64(double x) { return (unsigned)__double2loint(x); }
__device__ __forceinline__ unsigned umax(unsigned a, unsigned b) { return a > b ? a : b; }
// 2^lo <= x < 2^hi (false for a negative x and for NaN)
__device__ __forceinline__ bool in_pos(double x, int lo, int hi) { return hi64(x) - hi2(lo) < hi2(hi) - hi2(lo); }
// -2^hi < x <= -2^lo
__device__ __forceinline__ bool in_neg(double x, int lo, int hi) {
    return (hi64(x) ^ 0x80000000u) - hi2(lo) < hi2(hi) - hi2(lo);
}
// x = +-0 or 2^lo <= |x| < 2^hi
__device__ __forceinline__ bool in_mag(double x, int lo, int hi) {
    const unsigned n = habs(x);
    return (n - hi2(lo) < hi2(hi) - hi2(lo)) | ((n | lo64(x)) == 0u);
}
// a numerator that its quotient's residual can be exact for
__device__ __forceinline__ bool num_ok(double x) { return in_mag(x, -960, 200); }
// the sum of two quotients with the numerators n1, n2: large enough that what
// an underflowing residual loses is lost in its rounding too, or both zero
__device__ __forceinline__ bool sum_ok(double s, double n1, double n2) {
    return (habs(s) - hi2(-900) < hi2(200) - hi2(-900)) | (((habs(n1) | habs(n2)) | lo64(n1) | lo64(n2)) == 0u);
}
// the low word of an all-ones mantissa
__device__ __forceinline__ bool not_ones(double b) { return lo64(b) != 0xFFFFFFFFu; }

// A positive divisor shared by several quotients.  over() is x / b where its
// test holds; ok collects the tests, and where one fails the caller divides
// again with the plain form.
struct Den64 {
    double b, y;
    bool ok;
};
__device__ __forceinline__ Den64 den64(double b) {
    return {b, inv64(b), in_pos(b, -60, 60) & not_ones(b)};
}
__device__ __forceinline__ double over(double x, const Den64 &d, bool &ok) {
    ok &= d.ok & num_ok(x);
    return quo(x, d.b, d.y);
}

// ---------------------------------------------------------------------------
// WENO-Z (weno of mhd_device.cuh, the same roundings).  Products by powers of
// two are exact, so they are folded into fused multiply-adds: with
// z = RN(2 vc - U10), RN(2 U10 - 4 vc) = -2 z, and a square of a doubled
// difference is four times the square of the difference.  HALF: the weights
// of a uniform axis, all exactly 1/2, for which U01 = RN(vc + vp1) / 2.  About
// 175 FP64 operations a variable against about 245 of the plain form.
// Returns whether the result stands.
// ---------------------------------------------------------------------------
// one side: P and B of its three candidates -> the face value; hb, lo collect
// the high words of the B (non-negative) and the low words of the divisors
__device__ __forceinline__ double wenoz64(double P1, double P2, double P3, double B1, double B2, double B3, unsigned &hb,
                                          unsigned &lo, unsigned &hq) {
    const double eps = 1.0e-40;
    const double g1 = 1.0 / 10.0, g2 = 6.0 / 10.0, g3 = 3.0 / 10.0;
    const double tau5 = fabs(B1 - B3);
    const double d1 = eps + B1, d2 = eps + B2, d3 = eps + B3;
    const double q1 = quo(tau5, d1, inv64(d1)), q2 = quo(tau5, d2, inv64(d2)), q3 = quo(tau5, d3, inv64(d3));
    const double w1 = g1 * (1.0 + q1 * q1), w2 = g2 * (1.0 + q2 * q2), w3 = g3 * (1.0 + q3 * q3);
    const double n = w1 * P1 + w2 * P2 + w3 * P3, s = w1 + w2 + w3;
    hb = umax(umax(hi64(B1), hi64(B2)), umax(hi64(B3), hb));
    lo = umax(umax(lo64(d1), lo64(d2)), umax(umax(lo64(d3), lo64(s)), lo));
    const double q = quo(n, s, inv64(s));
    hq = habs(q);
    return q;
}

template <bool HALF>
__device__ __forceinline__ bool weno64(const double *__restrict__ w, double vm2, double vm1, double vc, double vp1,
                                       double vp2, double &vm_out, double &vp_out) {
    const double r4 = 4.0 * (13.0 / 12.0);  // exact: 13/12 scaled
    double U01, U12, U10, U21, U00, U11;
    if (HALF) {
        U01 = 0.5 * (vc + vp1);
        U12 = 0.5 * (vp1 + vp2);
        U10 = 0.5 * (vm1 + vc);
        U21 = 0.5 * (vm2 + vm1);
        U00 = __fma_rn(0.5, vm1 - vm2, vm1);
        U11 = __fma_rn(0.5, vp1 - vp2, vp1);
    } else {
        U01 = w[0] * vc + w[1] * vp1;
        U12 = w[2] * vp1 + w[3] * vp2;
        U10 = w[4] * vm1 + w[5] * vc;
        U21 = w[6] * vm2 + w[7] * vm1;
        U00 = vm1 + w[8] * (vm1 - vm2);
        U11 = vp1 + w[9] * (vp1 - vp2);
    }
    const double c6 = 6.0 * vc;
    const double z10 = __fma_rn(2.0, vc, -U10), z01 = __fma_rn(2.0, vc, -U01);
    const double t4 = U01 - U10, t4s = t4 * t4;
    unsigned hb = 0u, lo = 0u, np, nm;
    {
        const double P1 = third64(__fma_rn(-2.0, U00, c6 - U10));
        const double P2 = third64(__fma_rn(2.0, U01, z10));
        const double P3 = third64(__fma_rn(2.0, U01 + vp1, -U12));
        const double a = U10 - U00, b = z10 - U00;
        const double B1 = r4 * (a * a) + b * b;
        const double t3 = U01 - z10;
        const double B2 = r4 * (t3 * t3) + t4s;
        const double t5 = __fma_rn(-2.0, vp1, U01) + U12;
        const double t6 = __fma_rn(-2.0, U12, __fma_rn(8.0, vp1, -(6.0 * U01)));
        const double B3 = __fma_rn(0.25, t6 * t6, r4 * (t5 * t5));
        vp_out = wenoz64(P1, P2, P3, B1, B2, B3, hb, lo, np);
    }
    {
        const double P1 = third64(__fma_rn(-2.0, U11, c6 - U01));
        const double P2 = third64(__fma_rn(2.0, U10, z01));
        const double P3 = third64(__fma_rn(2.0, U10 + vm1, -U21));
        const double a = U01 - U11, b = z01 - U11;
        const double B1 = r4 * (a * a) + b * b;
        const double t3 = U10 - z01;
        const double B2 = r4 * (t3 * t3) + t4s;
        const double t5 = __fma_rn(-2.0, vm1, U10) + U21;
        const double t6 = __fma_rn(-2.0, U21, __fma_rn(8.0, vm1, -(6.0 * U10)));
        const double B3 = __fma_rn(0.25, t6 * t6, r4 * (t5 * t5));
        vm_out = wenoz64(P1, P2, P3, B1, B2, B3, hb, lo, nm);
    }
    // every B below 2^100 (so nothing overflowed and the q are below 2^234;
    // a q too small for its quotient to round right leaves 1 + q^2 = 1), both
    // results large enough for the residual to be exact (the divisor is at
    // least 1), or every value zero
    const unsigned any = ((hi64(vm2) | hi64(vm1) | hi64(vc) | hi64(vp1) | hi64(vp2)) & 0x7FFFFFFFu) | lo64(vm2) |
                         lo64(vm1) | lo64(vc) | lo64(vp1) | lo64(vp2);
    const bool q_ok = (np - hi2(-960) < hi2(900) - hi2(-960)) & (nm - hi2(-960) < hi2(900) - hi2(-960));
    return (hb < hi2(100)) & (lo != 0xFFFFFFFFu) & (q_ok | (any == 0u));
}

// ---------------------------------------------------------------------------
// One face with HLLD: the face EOS, the signal speeds and hlld_lean of
// mhd_device.cuh with the same roundings.  Every divisor's reciprocal is
// formed once: rho serves p / rho and the three B^2 / rho of its side,
// sL - sM and sR - sM eight quotients each.  About 700 FP64 operations become
// about 480, in blocks of independent chains.
// Returns whether the result stands.
// ---------------------------------------------------------------------------
struct Side64 {
    double eps, cf, sq;  // internal energy, fast speed, sqrt(rho)
};
template <int DIR>
__device__ __forceinline__ Side64 side64(const double *p, double gm1, double ig, bool &ok) {
    using F = Frame<DIR>;
    Side64 s;
    const double rho = p[irho], pr = p[itau];
    const double ir = inv64(rho);
    s.eps = quo(quo(pr, rho, ir), gm1, ig);
    const double r2 = rho * rho;
    const double cs2 = s.eps * gm1 + quo(rho * gm1 * pr, r2, inv64(r2));
    const double cs = sqrt64(cs2);
    const double a2 = cs * cs;
    const double a4 = a2 * a2;
    const double b2n = quo(p[F::ibn] * p[F::ibn], rho, ir);
    const double b2t1 = quo(p[F::ibt1] * p[F::ibt1], rho, ir);
    const double b2t2 = quo(p[F::ibt2] * p[F::ibt2], rho, ir);
    const double b2 = b2n + b2t1 + b2t2;
    const double b4 = b2 * b2;
    const double disc = dmax((a4 + b4 + 2.0 * b2 * a2) - 4.0 * a2 * b2n, 0.0);
    s.cf = sqrt64(0.5 * (a2 + b2 + sqrt64(disc)));
    s.sq = sqrt64(rho);
    // density and pressure inside 2^-60 .. 2^60, so that the sound speed and
    // every quotient above stay normal; a B^2 / rho too small to round right
    // is lost beside the sound speed
    ok &= in_pos(rho, -60, 60) & not_ones(rho) & not_ones(r2) & in_pos(pr, -60, 60) & in_pos(disc, -400, 900);
    return s;
}

template <int DIR>
__device__ __forceinline__ bool hlld64(const double *pl, const double *pr, double gamma, double *fo) {
    using F = Frame<DIR>;
    constexpr int ivn = F::ivn, ivt1 = F::ivt1, ivt2 = F::ivt2, ibn = F::ibn, ibt1 = F::ibt1, ibt2 = F::ibt2;
    const double gm1 = gamma - 1.0, ig = inv64(gm1);
    bool ok = in_pos(gm1, -60, 60) & not_ones(gm1) & num_ok(pl[ibn]);
    const Side64 L = side64<DIR>(pl, gm1, ig, ok), R = side64<DIR>(pr, gm1, ig, ok);
    const double den = L.sq + R.sq, iden = inv64(den);
    const double ubar = quo(L.sq * pl[ivn] + R.sq * pr[ivn], den, iden);
    const double cbar = quo(L.sq * L.cf + R.sq * R.cf, den, iden);
    const double sL = dmin(pl[ivn] - L.cf, ubar - cbar);
    const double sR = dmax(pr[ivn] + R.cf, ubar + cbar);
    ok &= not_ones(den);
    if (sL >= 0.0 || sR <= 0.0) {
        double u[9];
        build_state<double, DIR>(sL >= 0.0 ? pl : pr, sL >= 0.0 ? L.eps : R.eps, u, fo);
        return ok;
    }
    const double b2L = pl[ibx] * pl[ibx] + pl[iby] * pl[iby] + pl[ibz] * pl[ibz];
    const double b2R = pr[ibx] * pr[ibx] + pr[iby] * pr[iby] + pr[ibz] * pr[ibz];
    const double pLt = pl[itau] + 0.5 * b2L, pRt = pr[itau] + 0.5 * b2R;
    const double cL = sL - pl[ivn], cR = sR - pr[ivn];
    const double mL = pl[irho] * cL, mR = pr[irho] * cR;
    // sstar_hllc (rsolver_module.f90:86-93)
    const double dm = pr[irho] * cR - pl[irho] * cL;
    const double nM = pr[irho] * pr[ivn] * cR - pl[irho] * pl[ivn] * cL + pLt - pRt + pr[ibn] * pr[ibn] - pl[ibn] * pl[ibn];
    const double sM = quo(nM, dm, inv64(dm));
    const double dL = sL - sM, dR = sR - sM;
    const double yL = inv64(dL), yR = inv64(dR);
    ok &= num_ok(nM) & in_pos(dm, -100, 100) & not_ones(dm) & in_neg(dL, -60, 60) & not_ones(dL) & in_pos(dR, -60, 60) &
          not_ones(dR);
    double usL[9], usR[9], pstL[9], pstR[9], zL1, zL2, zR1, zR2;
    {
        double ul[9], ur[9];
        cons_state<double>(pl, L.eps, ul);
        cons_state<double>(pr, R.eps, ur);
#pragma unroll
        for (int i = irho; i <= itau; ++i) {
            if (i == ivn) continue;  // the fan's velocity, below
            const double nl = ul[i] * cL, nr = ur[i] * cR;
            usL[i] = quo<false>(nl, dL, yL);
            usR[i] = quo(nr, dR, yR);
            if (i == ivt1) { zL1 = nl; zR1 = nr; }
            if (i == ivt2) { zL2 = nl; zR2 = nr; }
        }
    }
    const double sqL = sqrt64(usL[irho]), sqR = sqrt64(usR[irho]);
    double sstarL = sM - quo(fabs(pl[ibn]), sqL, inv64(sqL));
    double sstarR = sM + quo(fabs(pr[ibn]), sqR, inv64(sqR));
    ok &= in_pos(usL[irho], -60, 60) & in_pos(usR[irho], -60, 60) & not_ones(usL[irho]) & not_ones(usR[irho]) &
          not_ones(sqL) & not_ones(sqR);
    usL[ibn] = pl[ibn];
    usR[ibn] = pr[ibn];
    if (((sstarL - sL) < 1.0e-4 * (sM - sL)) || ((sstarR - sR) > -1.0e-4 * (sR - sM))) {
        const double flt1 = (pl[ivn] * pl[ibt1] - pl[ivt1] * pl[ibn]), frt1 = (pr[ivn] * pr[ibt1] - pr[ivt1] * pr[ibn]);
        const double flt2 = (pl[ivn] * pl[ibt2] - pl[ivt2] * pl[ibn]), frt2 = (pr[ivn] * pr[ibt2] - pr[ivt2] * pr[ibn]);
        const double ds = sR - sL, ids = inv64(ds);
        ok &= not_ones(ds);
        const double n1 = sR * pr[ibt1] - sL * pl[ibt1] - (frt1 - flt1), n2 = sR * pr[ibt2] - sL * pl[ibt2] - (frt2 - flt2);
        ok &= num_ok(n1) & num_ok(n2);
        usL[ibt1] = quo(n1, ds, ids);
        usL[ibt2] = quo(n2, ds, ids);
        usR[ibt1] = usL[ibt1];
        usR[ibt2] = usL[ibt2];
        sstarL = sM;
        sstarR = sM;
    } else {
        const double bb = pl[ibn] * pl[ibn];
        double fac = mL * dL - bb, y = inv64(fac), n = mL * cL - bb;
        ok &= in_pos(fac, -60, 200) & not_ones(fac) & num_ok(pl[ibt1] * n) & num_ok(pl[ibt2] * n);
        usL[ibt1] = quo(pl[ibt1] * n, fac, y);
        usL[ibt2] = quo(pl[ibt2] * n, fac, y);
        fac = mR * dR - bb;
        y = inv64(fac);
        n = mR * cR - bb;
        ok &= in_pos(fac, -60, 200) & not_ones(fac) & num_ok(pr[ibt1] * n) & num_ok(pr[ibt2] * n);
        usR[ibt1] = quo(pr[ibt1] * n, fac, y);
        usR[ibt2] = quo(pr[ibt2] * n, fac, y);
    }
    const double irL = inv64(usL[irho]), irR = inv64(usR[irho]);
    usL[ivn] = usL[irho] * sM;
    {
        const double n1 = usL[ibn] * usL[ibt1] - pl[ibn] * pl[ibt1], n2 = usL[ibn] * usL[ibt2] - pl[ibn] * pl[ibt2];
        usL[ivt1] = usL[ivt1] - quo<false>(n1, dL, yL);
        usL[ivt2] = usL[ivt2] - quo<false>(n2, dL, yL);
        ok &= sum_ok(usL[ivt1], zL1, n1) & sum_ok(usL[ivt2], zL2, n2);
    }
    usR[ivn] = usR[irho] * sM;
    {
        const double n1 = usR[ibn] * usR[ibt1] - pr[ibn] * pr[ibt1], n2 = usR[ibn] * usR[ibt2] - pr[ibn] * pr[ibt2];
        usR[ivt1] = usR[ivt1] - quo(n1, dR, yR);
        usR[ivt2] = usR[ivt2] - quo(n2, dR, yR);
        ok &= sum_ok(usR[ivt1], zR1, n1) & sum_ok(usR[ivt2], zR2, n2);
    }
    pstL[ivn] = sM;
    pstL[ivt1] = quo(usL[ivt1], usL[irho], irL);
    pstL[ivt2] = quo(usL[ivt2], usL[irho], irL);
    pstR[ivn] = sM;
    pstR[ivt1] = quo(usR[ivt1], usR[irho], irR);
    pstR[ivt2] = quo(usR[ivt2], usR[irho], irR);
    const double pLs = mL * (sM - pl[ivn]) + pLt;
    const double pRs = mR * (sM - pr[ivn]) + pRt;
    const double bdotuL = pl[ibx] * pl[ivx] + pl[iby] * pl[ivy] + pl[ibz] * pl[ivz];
    const double bdotusL = usL[ibx] * pstL[ivx] + usL[iby] * pstL[ivy] + usL[ibz] * pstL[ivz];
    const double nEL = (pLs * sM - pLt * pl[ivn]) - (bdotusL - bdotuL) * pl[ibn];
    usL[itau] = usL[itau] + quo<false>(nEL, dL, yL);
    const double bdotuR = pr[ibx] * pr[ivx] + pr[iby] * pr[ivy] + pr[ibz] * pr[ivz];
    const double bdotusR = usR[ibx] * pstR[ivx] + usR[iby] * pstR[ivy] + usR[ibz] * pstR[ivz];
    const double nER = (pRs * sM - pRt * pr[ivn]) - (bdotusR - bdotuR) * pr[ibn];
    usR[itau] = usR[itau] + quo(nER, dR, yR);
    // the side whose fan the face lies in; its flux and state are rebuilt here
    const bool left = (sstarL >= 0.0) || (!(sstarR <= 0.0) && (sM >= 0.0));
    const double *pS = left ? pl : pr;
    const double s = left ? sL : sR;
    const double *usS = left ? usL : usR;
    double uS[9], fS[9];
    build_state<double, DIR>(pS, left ? L.eps : R.eps, uS, fS);
    if (sstarL >= 0.0 || sstarR <= 0.0) {
#pragma unroll
        for (int i = 1; i <= 8; ++i) fo[i] = fS[i] + s * (usS[i] - uS[i]);
        return ok;
    }
    const double sqs = sqL + sqR;
    // 1 / (sqL + sqR), rounded: the numerator is a power of two
    const double ysq = inv64(sqs), fac_1 = quo(1.0, sqs, ysq);
    const double fac_2 = sign1(pl[ibn]);
    const double sqLR = sqrt64(usL[irho] * usR[irho]);
    ok &= not_ones(sqs);
    double pss[9], bss[9];
    pss[ivn] = sM;
    pss[ivt1] = fac_1 * (sqL * pstL[ivt1] + sqR * pstR[ivt1] + (usR[ibt1] - usL[ibt1]) * fac_2);
    pss[ivt2] = fac_1 * (sqL * pstL[ivt2] + sqR * pstR[ivt2] + (usR[ibt2] - usL[ibt2]) * fac_2);
    bss[ibt1] = fac_1 * (sqL * usR[ibt1] + sqR * usL[ibt1] + sqLR * (pstR[ivt1] - pstL[ivt1]) * fac_2);
    bss[ibt2] = fac_1 * (sqL * usR[ibt2] + sqR * usL[ibt2] + sqLR * (pstR[ivt2] - pstL[ivt2]) * fac_2);
    bss[ibn] = usS[ibn];
    const double bdotuss = bss[ibx] * pss[ivx] + bss[iby] * pss[ivy] + bss[ibz] * pss[ivz];
    double uss[9];
    uss[irho] = usS[irho];
    uss[ivn] = uss[irho] * pss[ivn];
    uss[ivt1] = uss[irho] * pss[ivt1];
    uss[ivt2] = uss[irho] * pss[ivt2];
    // usL - sqL (...) on the left, usR + sqR (...) on the right
    const double dtau = (left ? sqL : sqR) * ((left ? bdotusL : bdotusR) - bdotuss) * fac_2;
    uss[itau] = left ? usS[itau] - dtau : usS[itau] + dtau;
    uss[ibx] = bss[ibx];
    uss[iby] = bss[iby];
    uss[ibz] = bss[ibz];
    const double sst = left ? sstarL : sstarR;
#pragma unroll
    for (int i = 1; i <= 8; ++i) fo[i] = fS[i] + s * (usS[i] - uS[i]) + sst * (uss[i] - usS[i]);
    return ok;
}

}  // namespace cumc
