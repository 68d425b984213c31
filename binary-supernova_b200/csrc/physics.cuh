// physics.cuh -- WENO5-Z, cell pressure, face energy and HLLC for the FP64
// path.  Every expression keeps the reference's evaluation order
// (a+b+c == (a+b)+c, a*b*c == (a*b)*c, x^2 == x*x) and this translation unit
// family is compiled with -fmad=false, IEEE division and square root, so the
// results are bit-identical to the reference's CPU path.
#pragma once

#include "bsn_internal.cuh"
#include "exact_div.cuh"

namespace bsn {
namespace f64 {

// WENO-Z nonlinear weights and the weighted sum (src/weno5.jl:14-21, 40, 60).
__device__ __forceinline__ double wenoz_sum(double b0, double b1, double b2, double d0, double d1, double d2,
                                            double q0, double q1, double q2) {
    const double eps = 1e-36;
    double tau5 = fabs(b0 - b2);
    double a0 = d0 * (1.0 + sq(tau5 / (eps + b0)));
    double a1 = d1 * (1.0 + sq(tau5 / (eps + b1)));
    double a2 = d2 * (1.0 + sq(tau5 / (eps + b2)));
    double asum = a0 + a1 + a2;
    double w0 = a0 / asum, w1 = a1 / asum, w2 = a2 / asum;
    return w0 * q0 + w1 * q1 + w2 * q2;
}

// Left- and right-biased WENO5-Z values at the interface between c2 and c3
// from the six cells c0..c5 (src/weno5.jl:25-61).  The right reconstruction's
// first two candidate polynomials and its first smoothness indicator are the
// same expressions on the same cells as the left's q1, q2 and beta1, and the
// 13/12 term of left beta2 equals that of right beta1, so they are computed
// once; the values are unchanged bit for bit.
__device__ __forceinline__ void weno5_lr(double c0, double c1, double c2, double c3, double c4, double c5,
                                         double* L, double* R) {
    const double t13 = 1.0 / 3.0, m76 = -7.0 / 6.0, e116 = 11.0 / 6.0, m16 = -1.0 / 6.0, f56 = 5.0 / 6.0;
    const double k1312 = 13.0 / 12.0, k14 = 1.0 / 4.0;
    double qA = t13 * c0 + m76 * c1 + e116 * c2;   // left q0
    double qB = m16 * c1 + f56 * c2 + t13 * c3;    // left q1 == right q0
    double qC = t13 * c2 + f56 * c3 + m16 * c4;    // left q2 == right q1
    double qD = e116 * c3 + m76 * c4 + t13 * c5;   // right q2
    double bA = k1312 * sq(c0 - 2.0 * c1 + c2) + k14 * sq(c0 - 4.0 * c1 + 3.0 * c2);   // left b0
    double bB = k1312 * sq(c1 - 2.0 * c2 + c3) + k14 * sq(c1 - c3);                    // left b1 == right b0
    double s2 = k1312 * sq(c2 - 2.0 * c3 + c4);
    double bC = s2 + k14 * sq(3.0 * c2 - 4.0 * c3 + c4);                              // left b2
    double bD = s2 + k14 * sq(c2 - 4.0 * c3 + 3.0 * c4);                              // right b1
    double bE = k1312 * sq(c3 - 2.0 * c4 + c5) + k14 * sq(3.0 * c3 - 4.0 * c4 + c5);   // right b2
    *L = wenoz_sum(bA, bB, bC, 1.0 / 10.0, 6.0 / 10.0, 3.0 / 10.0, qA, qB, qC);
    *R = wenoz_sum(bB, bD, bE, 3.0 / 10.0, 6.0 / 10.0, 1.0 / 10.0, qB, qC, qD);
}

// src/euler3d.jl:86-90
__device__ __forceinline__ double cell_pressure(double r, double mx, double my, double mz, double E,
                                                double gm1) {
    r = jmax(r, 1e-30);
    double KE = 0.5 * (sq(mx) + sq(my) + sq(mz)) / r;
    return jmax(gm1 * (E - KE), 0.0);
}

// src/euler3d.jl:99-106
__device__ __forceinline__ double EL_from_P(double PL, double rL, double mxL, double myL, double mzL,
                                            double gm1) {
    double rp = jmax(rL, 1e-30);
    double m2 = sq(mxL) + sq(myL) + sq(mzL);
    double KE_raw = 0.5 * m2 / rp;
    double KE = jmin(KE_raw, 0.5 * rp * 1e4);
    return PL / gm1 + KE;
}

// HLLC along the normal (src/hllc.jl:17-165).  Inputs/outputs are in the
// rotated (normal, t1, t2) ordering.
__device__ __forceinline__ void hllc_normal(double rL, double mnL, double mt1L, double mt2L, double EL,
                                            double rR, double mnR, double mt1R, double mt2R, double ER,
                                            double g, double gm1, double F[5]) {
    if (rL <= 0.0) { rL = 1e-30; mnL = 0.0; mt1L = 0.0; mt2L = 0.0; EL = 0.0; }
    else           { rL = jmax(rL, 1e-30); }
    if (rR <= 0.0) { rR = 1e-30; mnR = 0.0; mt1R = 0.0; mt2R = 0.0; ER = 0.0; }
    else           { rR = jmax(rR, 1e-30); }

    double m2L = sq(mnL) + sq(mt1L) + sq(mt2L);
    if (m2L > sq(rL) * 1e4) {
        double s = rL * 100.0 / sqrt(m2L);
        mnL *= s; mt1L *= s; mt2L *= s;
    }
    double m2R = sq(mnR) + sq(mt1R) + sq(mt2R);
    if (m2R > sq(rR) * 1e4) {
        double s = rR * 100.0 / sqrt(m2R);
        mnR *= s; mt1R *= s; mt2R *= s;
    }
    double KE_L = jmin(0.5 * (sq(mnL) + sq(mt1L) + sq(mt2L)) / rL, 0.5 * rL * 1e4);
    double KE_R = jmin(0.5 * (sq(mnR) + sq(mt1R) + sq(mt2R)) / rR, 0.5 * rR * 1e4);
    EL = jmax(EL, KE_L);
    ER = jmax(ER, KE_R);

    double vnL = mnL / rL, vt1L = mt1L / rL, vt2L = mt2L / rL;
    double vnR = mnR / rR, vt1R = mt1R / rR, vt2R = mt2R / rR;
    double pL = gm1 * (EL - KE_L);
    double pR = gm1 * (ER - KE_R);
    double csL = sqrt(g * pL / rL);
    double csR = sqrt(g * pR / rR);

    double SL, SR;
    if (pL > 0.0 && pR > 0.0) {
        double r_avg = 0.5 * (rL + rR);
        double cs_avg = 0.5 * (csL + csR);
        double p_star = jmax(0.0, 0.5 * (pL + pR) - 0.5 * (vnR - vnL) * r_avg * cs_avg);
        double gg = (g + 1.0) / (2.0 * g);
        double qL = p_star > pL ? sqrt(1.0 + gg * (p_star / pL - 1.0)) : 1.0;
        double qR = p_star > pR ? sqrt(1.0 + gg * (p_star / pR - 1.0)) : 1.0;
        SL = vnL - csL * qL;
        SR = vnR + csR * qR;
    } else {
        SL = jmin(vnL - csL, vnR - csR);
        SR = jmax(vnL + csL, vnR + csR);
    }

    double denom = rL * (SL - vnL) - rR * (SR - vnR);
    if (fabs(denom) < 1e-100) { F[0] = F[1] = F[2] = F[3] = F[4] = 0.0; return; }
    double S_star = (pR - pL + rL * vnL * (SL - vnL) - rR * vnR * (SR - vnR)) / denom;

    double FrL = mnL, FmnL = rL * sq(vnL) + pL, Fmt1L = mt1L * vnL, Fmt2L = mt2L * vnL;
    double FEL = (EL + pL) * vnL;
    if (SL >= 0.0) { F[0] = FrL; F[1] = FmnL; F[2] = Fmt1L; F[3] = Fmt2L; F[4] = FEL; return; }
    double FrR = mnR, FmnR = rR * sq(vnR) + pR, Fmt1R = mt1R * vnR, Fmt2R = mt2R * vnR;
    double FER = (ER + pR) * vnR;
    if (SR <= 0.0) { F[0] = FrR; F[1] = FmnR; F[2] = Fmt1R; F[3] = Fmt2R; F[4] = FER; return; }

    if (jmax(rL, rR) > 3.0 * jmin(rL, rR)) {
        double inv_dS = 1.0 / (SR - SL);
        double SLSR = SL * SR;
        F[0] = (SR * FrL - SL * FrR + SLSR * (rR - rL)) * inv_dS;
        F[1] = (SR * FmnL - SL * FmnR + SLSR * (mnR - mnL)) * inv_dS;
        F[2] = (SR * Fmt1L - SL * Fmt1R + SLSR * (mt1R - mt1L)) * inv_dS;
        F[3] = (SR * Fmt2L - SL * Fmt2R + SLSR * (mt2R - mt2L)) * inv_dS;
        F[4] = (SR * FEL - SL * FER + SLSR * (ER - EL)) * inv_dS;
        return;
    }
    if (S_star >= 0.0) {
        double dL = rL * (SL - vnL);
        double chi = dL / (SL - S_star);
        double EsL = fabs(dL) > 1e-100 ? chi * (EL / rL + (S_star - vnL) * (S_star + pL / dL)) : 0.0;
        F[0] = FrL + SL * (chi - rL);
        F[1] = FmnL + SL * (chi * S_star - mnL);
        F[2] = Fmt1L + SL * (chi * vt1L - mt1L);
        F[3] = Fmt2L + SL * (chi * vt2L - mt2L);
        F[4] = FEL + SL * (EsL - EL);
    } else {
        double dR = rR * (SR - vnR);
        double chi = dR / (SR - S_star);
        double EsR = fabs(dR) > 1e-100 ? chi * (ER / rR + (S_star - vnR) * (S_star + pR / dR)) : 0.0;
        F[0] = FrR + SR * (chi - rR);
        F[1] = FmnR + SR * (chi * S_star - mnR);
        F[2] = Fmt1R + SR * (chi * vt1R - mt1R);
        F[3] = Fmt2R + SR * (chi * vt2R - mt2R);
        F[4] = FER + SR * (EsR - ER);
    }
}

// One interface along direction d from six cells (rows of 5 conserved
// values plus the cell pressure): WENO of rho, m, P (clamped to [0, stencil
// max]), energy from P, rotated HLLC (src/gpu_kernels.jl:51-154,
// src/hllc.jl:176-208).  F is returned in (rho, mx, my, mz, E) order.
template <int D>
__device__ __forceinline__ void interface_flux(const double (&c)[6][6], double g, double gm1, double F[5]) {
    double L[5], R[5];
#pragma unroll
    for (int q = 0; q < 4; ++q) weno5_lr(c[0][q], c[1][q], c[2][q], c[3][q], c[4][q], c[5][q], &L[q], &R[q]);
    double PL, PR;
    weno5_lr(c[0][5], c[1][5], c[2][5], c[3][5], c[4][5], c[5][5], &PL, &PR);
    double PmaxL = jmax(jmax(jmax(jmax(c[0][5], c[1][5]), c[2][5]), c[3][5]), c[4][5]);
    double PmaxR = jmax(jmax(jmax(jmax(c[1][5], c[2][5]), c[3][5]), c[4][5]), c[5][5]);
    PL = jclamp(PL, 0.0, PmaxL);
    PR = jclamp(PR, 0.0, PmaxR);
    double EL = EL_from_P(PL, L[0], L[1], L[2], L[3], gm1);
    double ER = EL_from_P(PR, R[0], R[1], R[2], R[3], gm1);
    double Fr[5];
    if (D == 0) {
        hllc_normal(L[0], L[1], L[2], L[3], EL, R[0], R[1], R[2], R[3], ER, g, gm1, Fr);
        F[0] = Fr[0]; F[1] = Fr[1]; F[2] = Fr[2]; F[3] = Fr[3]; F[4] = Fr[4];
    } else if (D == 1) {
        hllc_normal(L[0], L[2], L[1], L[3], EL, R[0], R[2], R[1], R[3], ER, g, gm1, Fr);
        F[0] = Fr[0]; F[1] = Fr[2]; F[2] = Fr[1]; F[3] = Fr[3]; F[4] = Fr[4];
    } else {
        hllc_normal(L[0], L[3], L[1], L[2], EL, R[0], R[3], R[1], R[2], ER, g, gm1, Fr);
        F[0] = Fr[0]; F[1] = Fr[2]; F[2] = Fr[3]; F[3] = Fr[1]; F[4] = Fr[4];
    }
}

// hm2 / r, IEEE-rounded: the kinetic energy of a cell (hm2 = 0.5 m^2).  Gas at
// rest, the most common cell of an atmosphere, needs no division.
__device__ __forceinline__ double kinetic(double hm2, double r) {
    if (abs_hi(r) - hi_pow2(-100) < hi_pow2(116) - hi_pow2(-100) && r > 0.0 && abs_hi(hm2) < hi_pow2(240)) {
        if (hm2 == 0.0) return 0.0;
        if (!too_small(hm2, kNumRhoLo)) return quot_pos(hm2, r, recip_rn(r));
    }
    return hm2 / r;
}

// Density/pressure floors (src/gpu_kernels.jl:26-46).  Pfl_gm1 = P_floor/(gamma-1).
__device__ __forceinline__ void apply_floor(double& r, double& mx, double& my, double& mz, double& E,
                                            double rho_floor, double P_floor, double Pfl_gm1, double gm1) {
    if (r < rho_floor) {
        r = rho_floor; mx = 0.0; my = 0.0; mz = 0.0; E = Pfl_gm1;
    } else {
        double KE = kinetic(0.5 * (sq(mx) + sq(my) + sq(mz)), r);
        double P = gm1 * (E - KE);
        if (P < P_floor) E = Pfl_gm1 + KE;
    }
}

// ---------------------------------------------------------------------------
// The same interface for ordinary data (every cell below 2^116 in magnitude,
// so nothing overflows and no NaN arises): the same operations in the same
// order, with the divisions by shared reciprocals (exact_div.cuh) and plain
// comparisons where the reference's max / min propagate NaN.  The bits are
// interface_flux's; operands outside quot's range are reported instead.

// wenoz_sum with y_k = RN(1 / (1e-36 + b_k)), e_k = 1e-36 + b_k
__device__ __forceinline__ double wenoz_sum_ord(double b0, double b2, double e0, double e1, double e2, double y0,
                                                double y1, double y2, double d0, double d1, double d2, double q0,
                                                double q1, double q2) {
    const double tau5 = fabs(b0 - b2);
    const double a0 = d0 * (1.0 + sq(quot_pos(tau5, e0, y0)));
    const double a1 = d1 * (1.0 + sq(quot_pos(tau5, e1, y1)));
    const double a2 = d2 * (1.0 + sq(quot_pos(tau5, e2, y2)));
    const double asum = a0 + a1 + a2;
    const double ys = recip_rn(asum);
    return quot_pos(a0, asum, ys) * q0 + quot_pos(a1, asum, ys) * q1 + quot_pos(a2, asum, ys) * q2;
}

__device__ __forceinline__ void weno5_lr_ord(double c0, double c1, double c2, double c3, double c4, double c5,
                                             double* L, double* R) {
    const double t13 = 1.0 / 3.0, m76 = -7.0 / 6.0, e116 = 11.0 / 6.0, m16 = -1.0 / 6.0, f56 = 5.0 / 6.0;
    const double k1312 = 13.0 / 12.0, k14 = 1.0 / 4.0, eps = 1e-36;
    const double qA = t13 * c0 + m76 * c1 + e116 * c2;
    const double qB = m16 * c1 + f56 * c2 + t13 * c3;
    const double qC = t13 * c2 + f56 * c3 + m16 * c4;
    const double qD = e116 * c3 + m76 * c4 + t13 * c5;
    const double bA = k1312 * sq(c0 - 2.0 * c1 + c2) + k14 * sq(c0 - 4.0 * c1 + 3.0 * c2);
    const double bB = k1312 * sq(c1 - 2.0 * c2 + c3) + k14 * sq(c1 - c3);
    const double s2 = k1312 * sq(c2 - 2.0 * c3 + c4);
    const double bC = s2 + k14 * sq(3.0 * c2 - 4.0 * c3 + c4);
    const double bD = s2 + k14 * sq(c2 - 4.0 * c3 + 3.0 * c4);
    const double bE = k1312 * sq(c3 - 2.0 * c4 + c5) + k14 * sq(3.0 * c3 - 4.0 * c4 + c5);
    const double eA = eps + bA, eB = eps + bB, eC = eps + bC, eD = eps + bD, eE = eps + bE;
    const double yB = recip_rn(eB);
    *L = wenoz_sum_ord(bA, bC, eA, eB, eC, recip_rn(eA), yB, recip_rn(eC), 1.0 / 10.0, 6.0 / 10.0, 3.0 / 10.0, qA, qB,
                       qC);
    *R = wenoz_sum_ord(bB, bE, eB, eD, eE, yB, recip_rn(eD), recip_rn(eE), 3.0 / 10.0, 6.0 / 10.0, 1.0 / 10.0, qB, qC,
                       qD);
}

// One side of hllc_normal up to its physical flux, with the density's
// reciprocal shared by its six quotients.
struct HllcSide {
    double r, y, mn, mt1, mt2, E, vn, vt1, vt2, p, cs;
};
__device__ __forceinline__ bool hllc_side_ord(HllcSide& s, double r, double y, double mn, double mt1, double mt2,
                                              double E, double g, double gm1) {
    bool bad = false;
    if (r <= 0.0) { r = 1e-30; mn = 0.0; mt1 = 0.0; mt2 = 0.0; E = 0.0; }
    else          { r = r > 1e-30 ? r : 1e-30; }
    double m2 = sq(mn) + sq(mt1) + sq(mt2);
    if (m2 > sq(r) * 1e4) {
        const double f = r * 100.0 / sqrt(m2);
        mn *= f; mt1 *= f; mt2 *= f;
        m2 = sq(mn) + sq(mt1) + sq(mt2);
    }
    const double hm2 = 0.5 * m2, cap = 0.5 * r * 1e4;
    double ke = quot_pos(hm2, r, y);
    s.vn = quot(mn, r, y); s.vt1 = quot(mt1, r, y); s.vt2 = quot(mt2, r, y);
    // the stencils leave momenta that fall off to the smallest doubles ahead
    // of every front: common enough to be divided here instead of sending the
    // face (and with it the warp) to the general code
    if (too_small(hm2, kNumRhoLo) | too_small(mn, kNumRhoLo) | too_small(mt1, kNumRhoLo) |
        too_small(mt2, kNumRhoLo)) {
        ke = hm2 / r;
        s.vn = mn / r; s.vt1 = mt1 / r; s.vt2 = mt2 / r;
    }
    const double KE = ke < cap ? ke : cap;
    E = E > KE ? E : KE;
    s.p = gm1 * (E - KE);
    const double gp = g * s.p;
    bad |= too_small(gp, kNumRhoLo) | too_small(E, kNumRhoLo);
    s.cs = sqrt(quot_pos(gp, r, y));
    s.r = r; s.y = y; s.mn = mn; s.mt1 = mt1; s.mt2 = mt2; s.E = E;
    return bad;
}

// hllc_normal; rL, rR's reciprocals yL, yR are those of max(r, 1e-30).
// Returns true when an operand left quot's range (F is then meaningless).
__device__ __forceinline__ bool hllc_normal_ord(double rL, double yL, double mnL, double mt1L, double mt2L, double EL,
                                                double rR, double yR, double mnR, double mt1R, double mt2R, double ER,
                                                double g, double gm1, double gg, double F[5]) {
    HllcSide A, B;
    bool bad = hllc_side_ord(A, rL, yL, mnL, mt1L, mt2L, EL, g, gm1);
    bad |= hllc_side_ord(B, rR, yR, mnR, mt1R, mt2R, ER, g, gm1);
    double SL, SR;
    if (A.p > 0.0 && B.p > 0.0) {
        const double r_avg = 0.5 * (A.r + B.r);
        const double cs_avg = 0.5 * (A.cs + B.cs);
        const double ps = 0.5 * (A.p + B.p) - 0.5 * (B.vn - A.vn) * r_avg * cs_avg;
        const double p_star = ps > 0.0 ? ps : 0.0;
        double qL = 1.0, qR = 1.0;
        if (p_star > A.p) {
            bad |= bad_denominator(A.p);
            qL = sqrt(1.0 + gg * (quot_pos(p_star, A.p, recip_rn(A.p)) - 1.0));
        }
        if (p_star > B.p) {
            bad |= bad_denominator(B.p);
            qR = sqrt(1.0 + gg * (quot_pos(p_star, B.p, recip_rn(B.p)) - 1.0));
        }
        SL = A.vn - A.cs * qL;
        SR = B.vn + B.cs * qR;
    } else {
        SL = jmin(A.vn - A.cs, B.vn - B.cs);
        SR = jmax(A.vn + A.cs, B.vn + B.cs);
    }

    const double denom = A.r * (SL - A.vn) - B.r * (SR - B.vn);
    if (fabs(denom) < 1e-100) { F[0] = F[1] = F[2] = F[3] = F[4] = 0.0; return bad; }
    const double snum = B.p - A.p + A.r * A.vn * (SL - A.vn) - B.r * B.vn * (SR - B.vn);
    bad |= bad_denominator(denom) | too_small(snum, kNumSpeedLo);
    const double S_star = quot(snum, denom, recip_rn(fabs(denom)));

    const double FrL = A.mn, FmnL = A.r * sq(A.vn) + A.p, Fmt1L = A.mt1 * A.vn, Fmt2L = A.mt2 * A.vn;
    const double FEL = (A.E + A.p) * A.vn;
    if (SL >= 0.0) { F[0] = FrL; F[1] = FmnL; F[2] = Fmt1L; F[3] = Fmt2L; F[4] = FEL; return bad; }
    const double FrR = B.mn, FmnR = B.r * sq(B.vn) + B.p, Fmt1R = B.mt1 * B.vn, Fmt2R = B.mt2 * B.vn;
    const double FER = (B.E + B.p) * B.vn;
    if (SR <= 0.0) { F[0] = FrR; F[1] = FmnR; F[2] = Fmt1R; F[3] = Fmt2R; F[4] = FER; return bad; }

    const double rmax = A.r > B.r ? A.r : B.r, rmin = A.r < B.r ? A.r : B.r;
    if (rmax > 3.0 * rmin) {
        const double inv_dS = 1.0 / (SR - SL);
        const double SLSR = SL * SR;
        F[0] = (SR * FrL - SL * FrR + SLSR * (B.r - A.r)) * inv_dS;
        F[1] = (SR * FmnL - SL * FmnR + SLSR * (B.mn - A.mn)) * inv_dS;
        F[2] = (SR * Fmt1L - SL * Fmt1R + SLSR * (B.mt1 - A.mt1)) * inv_dS;
        F[3] = (SR * Fmt2L - SL * Fmt2R + SLSR * (B.mt2 - A.mt2)) * inv_dS;
        F[4] = (SR * FEL - SL * FER + SLSR * (B.E - A.E)) * inv_dS;
        return bad;
    }
    // the star flux of the upwind side: one instance for both
    const bool left = S_star >= 0.0;
    const double S = left ? SL : SR, r = left ? A.r : B.r, y = left ? A.y : B.y, vn = left ? A.vn : B.vn;
    const double p = left ? A.p : B.p, E = left ? A.E : B.E;
    const double d = r * (S - vn), ds = S - S_star;
    bad |= bad_denominator(ds) | too_small(d, kNumSpeedLo);
    const double chi = quot(d, ds, recip_rn(fabs(ds)));
    double Es = 0.0;
    if (fabs(d) > 1e-100) {
        bad |= bad_denominator(d) | too_small(p, kNumSpeedLo);
        Es = chi * (quot_pos(E, r, y) + (S_star - vn) * (S_star + quot(p, d, recip_rn(fabs(d)))));
    }
    F[0] = (left ? FrL : FrR) + S * (chi - r);
    F[1] = (left ? FmnL : FmnR) + S * (chi * S_star - (left ? A.mn : B.mn));
    F[2] = (left ? Fmt1L : Fmt1R) + S * (chi * (left ? A.vt1 : B.vt1) - (left ? A.mt1 : B.mt1));
    F[3] = (left ? Fmt2L : Fmt2R) + S * (chi * (left ? A.vt2 : B.vt2) - (left ? A.mt2 : B.mt2));
    F[4] = (left ? FEL : FER) + S * (Es - E);
    return bad;
}

// EL_from_P with y = RN(1 / max(rL, 1e-30)) and igm1 = RN(1 / gm1)
__device__ __forceinline__ bool EL_from_P_ord(double PL, double rL, double y, double mxL, double myL, double mzL,
                                              double gm1, double igm1, double* E) {
    const double rp = rL > 1e-30 ? rL : 1e-30;
    const double hm2 = 0.5 * (sq(mxL) + sq(myL) + sq(mzL));
    double ke = quot_pos(hm2, rp, y);
    if (too_small(hm2, kNumRhoLo)) ke = hm2 / rp;
    const double cap = 0.5 * rp * 1e4;
    *E = quot_pos(PL, gm1, igm1) + (ke < cap ? ke : cap);
    return too_small(PL, kNumRhoLo);
}

// interface_flux along axis D (a constant, or at run time) for ordinary cells;
// gg = (g + 1) / (2 g), igm1 = RN(1 / gm1).  Returns true where the general
// interface_flux must be taken instead.
__device__ __forceinline__ bool interface_flux_ord(const double (&c)[6][6], double g, double gm1, double igm1,
                                                   double gg, int D, double F[5]) {
    double L[5], R[5], PL, PR;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        weno5_lr_ord(c[0][q], c[1][q], c[2][q], c[3][q], c[4][q], c[5][q], &L[q], &R[q]);
    weno5_lr_ord(c[0][5], c[1][5], c[2][5], c[3][5], c[4][5], c[5][5], &PL, &PR);
    // staged pressures are never negative or -0
    double Pm = c[1][5] > c[2][5] ? c[1][5] : c[2][5];
    Pm = Pm > c[3][5] ? Pm : c[3][5];
    Pm = Pm > c[4][5] ? Pm : c[4][5];
    PL = jclamp(PL, 0.0, Pm > c[0][5] ? Pm : c[0][5]);
    PR = jclamp(PR, 0.0, Pm > c[5][5] ? Pm : c[5][5]);
    const double yL = recip_rn(L[0] > 1e-30 ? L[0] : 1e-30), yR = recip_rn(R[0] > 1e-30 ? R[0] : 1e-30);
    double EL, ER;
    bool bad = EL_from_P_ord(PL, L[0], yL, L[1], L[2], L[3], gm1, igm1, &EL);
    bad |= EL_from_P_ord(PR, R[0], yR, R[1], R[2], R[3], gm1, igm1, &ER);
    // (normal, t1, t2) = (x, y, z), (y, x, z), (z, x, y)
    double Fr[5];
    bad |= hllc_normal_ord(L[0], yL, D == 0 ? L[1] : (D == 1 ? L[2] : L[3]), D == 0 ? L[2] : L[1],
                           D == 2 ? L[2] : L[3], EL, R[0], yR, D == 0 ? R[1] : (D == 1 ? R[2] : R[3]),
                           D == 0 ? R[2] : R[1], D == 2 ? R[2] : R[3], ER, g, gm1, gg, Fr);
    F[0] = Fr[0];
    F[1] = D == 0 ? Fr[1] : Fr[2];
    F[2] = D == 0 ? Fr[2] : (D == 1 ? Fr[1] : Fr[3]);
    F[3] = D == 2 ? Fr[1] : Fr[3];
    F[4] = Fr[4];
    return bad;
}

// interface_flux along axis D, out of line: the rare faces of interface_flux_ord
__device__ __noinline__ inline void general_flux(const double (&c)[6][6], double g, double gm1, int D, double F[5]) {
    if (D == 0) interface_flux<0>(c, g, gm1, F);
    else if (D == 1) interface_flux<1>(c, g, gm1, F);
    else interface_flux<2>(c, g, gm1, F);
}
// a gamma - 1 that quot can divide pressures by
__device__ __forceinline__ bool ordinary_gamma(double gm1) { return gm1 >= 0x1p-20 && gm1 < 0x1p20; }

// apply_floor (active cells) and cell_pressure of one cell with one division:
// both use the cell's kinetic energy.  Returns true when the cell is
// ordinary; the general code does the others.
__device__ __noinline__ inline void floor_and_pressure_general(double (&v)[5], bool act, double rho_floor, double P_floor,
                                                        double Pfl_gm1, double gm1, double* P) {
    if (act) apply_floor(v[0], v[1], v[2], v[3], v[4], rho_floor, P_floor, Pfl_gm1, gm1);
    *P = cell_pressure(v[0], v[1], v[2], v[3], v[4], gm1);
}
__device__ __forceinline__ bool floor_and_pressure(double (&v)[5], bool act, double rho_floor, double P_floor,
                                                   double Pfl_gm1, double gm1, double* P) {
    unsigned big = abs_hi(v[0]);
#pragma unroll
    for (int q = 1; q < 5; ++q) { const unsigned h = abs_hi(v[q]); big = h > big ? h : big; }
    const double hm2 = 0.5 * (sq(v[1]) + sq(v[2]) + sq(v[3]));
    if (big >= kCellHi || !(v[0] >= 1e-30) || (act && v[0] < rho_floor)) {
        floor_and_pressure_general(v, act, rho_floor, P_floor, Pfl_gm1, gm1, P);
        big = abs_hi(*P);
#pragma unroll
        for (int q = 0; q < 5; ++q) { const unsigned h = abs_hi(v[q]); big = h > big ? h : big; }
        return big < kCellHi;
    }
    double KE = quot_pos(hm2, v[0], recip_rn(v[0]));
    if (too_small(hm2, kNumRhoLo)) KE = hm2 / v[0];
    double p = gm1 * (v[4] - KE);
    if (act && p < P_floor) {
        v[4] = Pfl_gm1 + KE;
        p = gm1 * (v[4] - KE);
    }
    *P = p > 0.0 ? p : 0.0;
    return abs_hi(v[4]) < kCellHi && abs_hi(*P) < kCellHi;
}

// rotating_frame_source! (src/relax_ic.jl:150-176) on one cell's RHS d[5]:
// centrifugal rho Omega^2 (x, y) plus Coriolis 2 Omega (m_y, -m_x) on the
// momentum, rho v . a_centrifugal on the energy, in the reference's
// expression order.
__device__ __forceinline__ void rot_frame_src(double* d, double u0, double u1, double u2, double xc, double yc,
                                              double om) {
    const double O2 = om * om;
    d[1] = d[1] + (O2 * u0 * xc + 2.0 * om * u2);
    d[2] = d[2] + (O2 * u0 * yc - 2.0 * om * u1);
    d[4] = d[4] + O2 * (xc * u1 + yc * u2);
}

// relax_damping_source! (src/relax_ic.jl:59-120) on one cell's RHS d[5]:
// momentum damped toward the co-rotation velocity (-Omega y, Omega x, 0) over
// t_damp, the energy by the work of that force (inv_td = 1 / t_damp).
__device__ __forceinline__ void damp_src(double* d, double u0, double u1, double u2, double u3, double xc, double yc,
                                         double inv_td, double t_damp, double om) {
    const double rs = jmax(u0, 1e-30);
    if (om == 0.0) {
        d[1] = d[1] - u1 * inv_td;
        d[2] = d[2] - u2 * inv_td;
        d[3] = d[3] - u3 * inv_td;
        d[4] = d[4] - (u1 * u1 + u2 * u2 + u3 * u3) / (rs * t_damp);
    } else {
        const double vx = u1 / rs, vy = u2 / rs, vz = u3 / rs;
        const double vrotx = -om * yc, vroty = om * xc;
        const double vrx = vx - vrotx, vry = vy - vroty;
        d[1] = d[1] - rs * vrx * inv_td;
        d[2] = d[2] - rs * vry * inv_td;
        d[3] = d[3] - u3 * inv_td;
        d[4] = d[4] - rs * (vx * vrx + vy * vry + vz * vz) * inv_td;
    }
}

// CFL speed of one cell (src/gpu_kernels.jl:174-191).
__device__ __noinline__ inline double cfl_speed_general(double U0, double U1, double U2, double U3, double U4, double g,
                                                        double gm1, double idx, double idy, double idz) {
    double r = jmax(U0, 1e-30);
    double vx = U1 / r, vy = U2 / r, vz = U3 / r;
    double KE = 0.5 * (sq(vx) + sq(vy) + sq(vz));
    double P = jmax(gm1 * (U4 / r - KE) * r, 0.0);
    double cs = sqrt(g * P / r);
    return jmax(jmax((fabs(vx) + cs) * idx, (fabs(vy) + cs) * idy), (fabs(vz) + cs) * idz);
}
// ... the five quotients by the density from one reciprocal; cells outside
// quot's range take the general form.
__device__ __forceinline__ double cfl_speed(double U0, double U1, double U2, double U3, double U4, double g,
                                            double gm1, double idx, double idy, double idz) {
    unsigned big = abs_hi(U0);
    bool bad = !(U0 >= 1e-30);
    const double m[4] = {U1, U2, U3, U4};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const unsigned h = abs_hi(m[q]);
        big = h > big ? h : big;
        bad |= too_small(m[q], kNumRhoLo);
    }
    const double y = recip_rn(U0);
    const double vx = quot(U1, U0, y), vy = quot(U2, U0, y), vz = quot(U3, U0, y);
    const double KE = 0.5 * (sq(vx) + sq(vy) + sq(vz));
    const double p = gm1 * (quot(U4, U0, y) - KE) * U0;
    const double gp = g * (p > 0.0 ? p : 0.0);
    if (bad || big >= kCellHi || too_small(gp, kNumRhoLo) || abs_hi(gp) >= hi_pow2(600))
        return cfl_speed_general(U0, U1, U2, U3, U4, g, gm1, idx, idy, idz);
    const double cs = sqrt(quot_pos(gp, U0, y));
    const double sx = (fabs(vx) + cs) * idx, sy = (fabs(vy) + cs) * idy, sz = (fabs(vz) + cs) * idz;
    const double s = sx > sy ? sx : sy;
    return s > sz ? s : sz;
}

}  // namespace f64
}  // namespace bsn
