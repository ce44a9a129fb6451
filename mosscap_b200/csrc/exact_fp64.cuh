// Correctly rounded FP64 division and square root without branches, and the
// pointwise physics of physics.cuh written with them.
//
// The stage kernels spend most of their FP64 work on quotients and roots
// that must equal IEEE division and square root (bit-exact parity). The
// compiler's division ends each quotient in a branch to its special cases:
// measured on B200 at 20 warps per SM it takes the time of 16.6 FP64
// instructions per quotient (16.3 per root), whether one or five independent
// quotients are in flight, since nothing moves across the branch. The forms here
// are straight-line code for operands whose exponents were checked
// beforehand, once per cell (the range tests below) instead of once per
// quotient: 9 FP64 instructions per quotient, 5 for a further quotient with
// the same denominator, 8 per root, all of them free to overlap.
//
// Where a product with a power of two feeds an addition the two are written
// as one fma: the product is exact, so the result is the same rounding of the
// same sum as in physics.cuh. Everything else keeps the order of
// physics.cuh, whose functions are evaluated instead (generic form) wherever
// a range test fails. Measured (B200, two steps, bit-identical): KH 2048^2 WENO5-Z
// + HLLC 3.76 -> 3.16 ms, KH 256^2 (8 steps) 1.05 -> 0.80 ms, 384 MUSCL + HLLC
// problems (4 steps) 10.4 -> 9.5 ms.
//
// Division (Markstein, IBM J. Res. Dev. 34, 1990; Cornea, Harrison and Tang,
// "Scientific Computing on Itanium-based Systems", 2002): the seed
// rcp.approx.ftz.f64 (relative error <= 2^-19.9 over all of its inputs,
// measured; it reads the operand's upper word only) is refined by two
// Newton steps to y2 = RN((1/b)(1 + z)), |z| <= 2^-79; the quotient is corrected
// once with the half-refined reciprocal, which leaves it within
// (1/2 + 2^-26) ulp of a/b, and once more with y2, where the residual is exact.
// The last rounding could only differ from RN(a/b) if a/b lay within
// ulp/2 * |y2 b - 1| of a rounding boundary. For 53-bit integers A, B (the
// operands' significands) a quotient that is not on one is at least 1/(2B) ulp
// away from it, so that needs B > 2^53 (1 - 2^-27) and 1/b within |z| of a
// rounding boundary of its own. For those B the seed is the same, 1/2 exactly
// (scaled), the first step leaves an error below 2^-53 and the second |z| <= 2^-105,
// which leaves B = 2^53 - 1 alone (M = 2^53 + 1, M B = 2^106 - 1): its reciprocal
// lies just above a boundary and y2 on it, where rounding to even goes down. The
// lowest bit of e1 is set for that one (2^-52 of a correction that is itself
// below 2^-39). Tested on the closest quotients of every B = 2^53 - k, odd
// k < 2^15 (tests/test_exact_ops_gpu.py).
//
// Square root (same sources; Cornea-Hasegan, Golliver and Markstein, ARITH-14,
// 1999, for the enumeration of the hard cases): seed rsqrt.approx.ftz.f64
// (<= 2^-20.0), one third-order step for root and half reciprocal, one exact
// residual. The value before the last rounding is within 2^-102.8 of the root of
// x in [1, 4); a root at odd distance j from a rounding boundary, in units where
// the boundary's square is an integer, is at least j 2^-108 from it, so only
// j <= 37 can round differently; all significands with j < 64 are tested.
#pragma once

#include "physics.cuh"

namespace mc {

__device__ __forceinline__ double rcp_seed(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    return r;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

// 1 / b for exact_quot: y1 within 2^-39 of it, y2 within an ulp.
struct Recip {
    double b, y1, y2;
};
__device__ __forceinline__ Recip recip_of(double b) {
    Recip r;
    r.b = b;
    const double y0 = rcp_seed(b);
    const double e0 = fma(-b, y0, 1.0);
    r.y1 = fma(y0, e0, y0);
    double e1 = fma(-b, r.y1, 1.0);
    e1 = __hiloint2double(__double2hiint(e1), __double2loint(e1) | 1);
    r.y2 = fma(r.y1, e1, r.y1);
    return r;
}

// RN(a / b) for b whose reciprocal is normal, and a that is zero (b > 0 then:
// the residuals are formed as b q - a, which keeps the zero's sign) or so that
// the quotient is normal and |a| > 2^-900.
__device__ __forceinline__ double exact_quot(double a, const Recip& r) {
    double q = __dmul_rn(a, r.y1);
    double d = fma(r.b, q, -a);
    q = fma(-d, r.y1, q);
    d = fma(r.b, q, -a);
    return fma(-d, r.y2, q);
}
__device__ __forceinline__ double exact_div(double a, double b) {
    return exact_quot(a, recip_of(b));
}
// RN(1 / b)
__device__ __forceinline__ double exact_rcp(double b) {
    const Recip r = recip_of(b);
    const double d = fma(b, r.y2, -1.0);
    return fma(-d, r.y2, r.y2);
}

// RN(sqrt(x)) for x in [2^-900, 2^900]. Anything else gives no such value and
// no fault (negative x: NaN).
__device__ __forceinline__ double exact_sqrt(double x) {
    const double y0 = rsqrt_seed(x);
    double g = __dmul_rn(x, y0);
    double h = __hiloint2double(__double2hiint(y0) - 0x00100000, __double2loint(y0));  // y0 / 2
    const double e = fma(-g, h, 0.5);
    const double c = fma(__dmul_rn(1.5, e), e, e);
    g = fma(g, c, g);
    h = fma(h, c, h);
    const double d = fma(-g, g, x);
    return fma(d, h, g);
}

// ---- Range tests -------------------------------------------------------------
//
// A cell is in range when rho and p lie in [2^-120, 2^100) and each velocity
// and mass fraction is zero or of magnitude in [2^-250, 2^100). Then every
// division and root below meets its conditions: sums and products of such
// values that are not zero are at least 2^-303 (an operand's last bit), WENO
// weights at least 1 and at most 2^650, and so on; the face states a
// reconstruction makes of them are tested again before the Riemann solver
// (positivity is not kept by it). Upper words as integers: one or two
// instructions of the integer pipe for each value, none of the FP64 pipe.
__device__ __forceinline__ bool in_range_pos(double x) {
    return (unsigned)(__double2hiint(x) - 0x38700000) < 0x46300000u - 0x38700000u;
}
__device__ __forceinline__ bool in_range_any(double x) {
    const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return hi - 0x30500000u < 0x46300000u - 0x30500000u || (hi | (unsigned)__double2loint(x)) == 0u;
}
// Four upper words of positive values at once.
__device__ __forceinline__ bool in_range_pos4(double a, double b, double c, double d) {
    const int ha = __double2hiint(a), hb = __double2hiint(b), hc = __double2hiint(c), hd = __double2hiint(d);
    return min(min(ha, hb), min(hc, hd)) >= 0x38700000 && max(max(ha, hb), max(hc, hd)) < 0x46300000;
}

// The constants of the gas of one launch, formed on the host (kernel
// parameters: constant-bank operands, no registers).
struct FastGas {
    double gm1, gfac;  // gamma - 1, (gamma + 1) / (2 gamma)
    double rgm1;       // RN(1 / (gamma - 1))
    int ok;            // gamma and gamma - 1 in [2^-20, 2^20]
};
inline FastGas fast_gas(double gamma) {
    FastGas g;
    g.gm1 = gamma - 1.0;
    g.gfac = (gamma + 1.0) / (2.0 * gamma);
    g.rgm1 = 1.0 / g.gm1;
    g.ok = gamma <= 0x1p20 && g.gm1 >= 0x1p-20 ? 1 : 0;
    return g;
}

// ---- physics.cuh's functions for values in range -------------------------------

// prim_from_cons; false: the cell is out of range and w holds no result.
template <int NDIM>
__device__ __forceinline__ bool fast_prim(double gm1, const double* q, double* w) {
    const Recip r = recip_of(q[0]);
    w[0] = q[0];
    w[1] = exact_quot(q[1], r);
    bool ok = in_range_pos(q[0]) && in_range_any(w[1]);
    double v2 = __dmul_rn(w[1], w[1]);
    if constexpr (NDIM > 1) {
        w[2] = exact_quot(q[2], r);
        v2 = __dadd_rn(v2, __dmul_rn(w[2], w[2]));
        ok = ok && in_range_any(w[2]);
    }
    if constexpr (NDIM > 2) {
        w[3] = exact_quot(q[3], r);
        v2 = __dadd_rn(v2, __dmul_rn(w[3], w[3]));
        ok = ok && in_range_any(w[3]);
    }
    // E - (0.5 rho) v2: the factor 1/2 is exact
    w[1 + NDIM] = __dmul_rn(gm1, fma(-0.5, __dmul_rn(q[0], v2), q[1 + NDIM]));
    return ok && in_range_pos(w[1 + NDIM]);
}

// cfl_dt of a cell in range.
template <int NDIM>
__device__ __forceinline__ double fast_cfl_dt(double gamma, double dx, const double* w) {
    const double cs = exact_sqrt(exact_div(__dmul_rn(gamma, w[1 + NDIM]), w[0]));
    double v2 = __dmul_rn(w[1], w[1]);
    if constexpr (NDIM > 1) {
        v2 = __dadd_rn(v2, __dmul_rn(w[2], w[2]));
    }
    if constexpr (NDIM > 2) {
        v2 = __dadd_rn(v2, __dmul_rn(w[3], w[3]));
    }
    const double vel = v2 == 0.0 ? 0.0 : exact_sqrt(v2);
    return exact_div(dx, __dadd_rn(cs, vel));
}

// min of two finite non-negative doubles (their bits order as integers): the
// integer pipe's comparison in place of an FP64 one.
__device__ __forceinline__ double min_nonneg(double a, double b) {
    const unsigned long long x = (unsigned long long)__double_as_longlong(a);
    const unsigned long long y = (unsigned long long)__double_as_longlong(b);
    return __longlong_as_double((long long)(y < x ? y : x));
}
__device__ __forceinline__ bool same_sign(double a, double b) {
    return (__double2hiint(a) ^ __double2hiint(b)) >= 0;
}

// Half of limited_slope for finite arguments: the sign factors 0 and +-1 are
// selections instead of sums and products (0 * min is +0 here).
template <int LIM>
__device__ __forceinline__ double fast_half_slope(double um, double up) {
    if constexpr (LIM == kVanLeer) {
        const double p = um * up;
        return p > 0.0 ? exact_div(p, um + up) : 0.0;
    } else if constexpr (LIM == kMonotonizedCentral) {
        const double m = min_nonneg(fabs(um), min_nonneg(fabs(0.25 * (um + up)), fabs(up)));
        return same_sign(um, up) ? copysign(m, um) : 0.0;
    } else {
        const double m = 0.5 * min_nonneg(fabs(um), fabs(up));
        return same_sign(um, up) ? copysign(m, um) : 0.0;
    }
}

// reconstruct for a stencil in range.
template <int REC, int LIM>
__device__ __forceinline__ void fast_reconstruct(const double* s, double& wl, double& wr) {
    const double c = s[2];
    if constexpr (REC == kFog) {
        wl = c;
        wr = c;
    } else if constexpr (REC == kMuscl) {
        const double h = fast_half_slope<LIM>(c - s[1], s[3] - c);
        wl = c - h;
        wr = c + h;
    } else if constexpr (REC == kPpm) {
        const double um = s[1] - s[0], u0 = c - s[1], u1 = s[3] - c, up = s[4] - s[3];
        // half slopes: the factor 2 goes into 1/6 (exact)
        const double hm = fast_half_slope<LIM>(um, u0);
        const double h0 = fast_half_slope<LIM>(u0, u1);
        const double hp = fast_half_slope<LIM>(u1, up);
        const double k = 2.0 * (1.0 / 6.0);
        double l = fma(0.5, s[1] + c, -(k * (h0 - hm)));
        double r = fma(0.5, c + s[3], -(k * (hp - h0)));
        if ((r - c) * (c - l) <= 0.0) {
            l = c;
            r = c;
        }
        const double c3 = 3.0 * c;
        if (fabs(r - c) >= 2.0 * fabs(l - c)) {
            r = fma(-2.0, l, c3);
        }
        if (fabs(l - c) >= 2.0 * fabs(r - c)) {
            l = fma(-2.0, r, c3);
        }
        wl = l;
        wr = r;
    } else {
        // 71 FP64 instructions beside the five quotients (84 as written in
        // physics.cuh), the quotients independent of one another in two groups
        const double b_a = 13.0 / 12.0;
        const double eps = Consts<double>::weno_eps;
        const double c3 = 3.0 * c, c5 = 5.0 * c, c11 = 11.0 * c;
        const double d0 = fma(-2.0, s[1], s[0]) + c;
        const double d1 = fma(-2.0, c, s[1]) + s[3];
        const double d2 = fma(-2.0, s[3], c) + s[4];
        const double g0 = fma(-4.0, s[1], s[0]) + c3;
        const double g1 = s[1] - s[3];
        const double g2 = fma(-4.0, s[3], c3) + s[4];
        const double beta0 = fma(0.25, g0 * g0, b_a * (d0 * d0));
        const double beta1 = fma(0.25, g1 * g1, b_a * (d1 * d1));
        const double beta2 = fma(0.25, g2 * g2, b_a * (d2 * d2));
        const double tau5 = fabs(beta0 - beta2);
        // a tau5 too small for an exact residual leaves 1 + ind^2 = 1 in any case
        const double ind0 = exact_div(tau5, beta0 + eps);
        const double ind1 = exact_div(tau5, beta1 + eps);
        const double ind2 = exact_div(tau5, beta2 + eps);
        const double j0 = ind0 * ind0 + 1.0;
        const double j1 = 6.0 * (ind1 * ind1 + 1.0);
        const double j2 = ind2 * ind2 + 1.0;
        {
            const double e0 = fma(2.0, c, 5.0 * s[1]) - s[0];
            const double e1 = fma(2.0, s[1], c5 - s[3]);
            const double e2 = c11 + fma(2.0, s[4], -(7.0 * s[3]));
            const double a0 = 3.0 * j0;
            const double den = 6.0 * (a0 + j1 + j2);
            wl = exact_div(e2 * j2 + (e1 * j1 + e0 * a0), den);
        }
        {
            const double e0 = fma(2.0, c, 5.0 * s[3]) - s[4];
            const double e1 = fma(2.0, s[3], c5 - s[1]);
            const double e2 = c11 + fma(2.0, s[0], -(7.0 * s[1]));
            const double a0 = 3.0 * j2;
            const double den = 6.0 * (a0 + j1 + j0);
            wr = exact_div(e2 * j0 + (e1 * j1 + e0 * a0), den);
        }
    }
}

// riemann; false: a face state is out of range and flux holds no result.
template <int RS, int NDIM>
__device__ __forceinline__ bool fast_riemann(double gamma, const FastGas& gas, int axis, const double* wL,
                                             const double* wR, double* flux) {
    constexpr int nh = 2 + NDIM;
    constexpr int ie = 1 + NDIM;
    const double tiny = 1e-20;
    const double vL = along<NDIM>(wL, axis);
    const double vR = along<NDIM>(wR, axis);
    const double pL = wL[ie], pR = wR[ie];
    bool ok = in_range_pos4(wL[0], wR[0], pL, pR);
    const double csL = exact_sqrt(exact_div(gamma * pL, wL[0]));
    const double csR = exact_sqrt(exact_div(gamma * pR, wR[0]));
    // cons_from_prim: momenta and total energy (0.5 rho v^2 with an exact 1/2)
    double qL[nh], qR[nh];
    double kL = 0.0, kR = 0.0;
    qL[0] = wL[0];
    qR[0] = wR[0];
#pragma unroll
    for (int d = 1; d <= NDIM; ++d) {
        qL[d] = wL[0] * wL[d];
        qR[d] = wR[0] * wR[d];
        kL = d == 1 ? wL[d] * wL[d] : kL + wL[d] * wL[d];
        kR = d == 1 ? wR[d] * wR[d] : kR + wR[d] * wR[d];
    }
    const Recip rg{gas.gm1, gas.rgm1, gas.rgm1};
    qL[ie] = fma(0.5, wL[0] * kL, exact_quot(pL, rg));
    qR[ie] = fma(0.5, wR[0] * kR, exact_quot(pR, rg));
    if constexpr (RS == kHllc) {
        const double cs2 = csL + csR, rho2 = wL[0] + wR[0];
        // (vL - vR) rho_avg cs_avg with both factors 1/2 taken out (exact)
        const double p_mid = 0.5 * fma(0.25, (vL - vR) * rho2 * cs2, pL + pR);
        // used only where p_mid > p: the quotient is then at least 1, the root's argument too
        const double sqL = exact_sqrt(gas.gfac * (exact_div(p_mid, pL) - 1.0) + 1.0);
        const double sqR = exact_sqrt(gas.gfac * (exact_div(p_mid, pR) - 1.0) + 1.0);
        const double cLstar = (p_mid <= pL) ? 1.0 : sqL;
        const double cRstar = (p_mid <= pR) ? 1.0 : sqR;
        const double aL = vL - csL * cLstar;
        const double aR = vR + csR * cRstar;
        const double bM = smin(-tiny, aL);
        const double bP = smax(tiny, aR);
        double vxL = vL - aL;
        double vxR = vR - aR;
        const double tL = pL + vxL * along<NDIM>(qL, axis);
        const double tR = pR + vxR * along<NDIM>(qR, axis);
        const double mL = wL[0] * vxL;
        const double mR = -(wR[0] * vxR);
        const Recip rm = recip_of(mL + mR);
        const double aM = exact_quot(tL - tR, rm);
        const double cp = smax(exact_quot(mL * tR + mR * tL, rm), 0.0);
        // the upwind side only: the other's flux has weight zero. For finite g
        // s f + 0 g is s f, but for the sign of a zero, and no result depends on
        // that: every flux difference is added to a sum that starts from +0
        const bool left = aM >= 0.0;
        const double den = left ? (aM - bM) : (bP - aM);
        const Recip rd = recip_of(den);
        const double s_out = exact_quot(left ? aM : -aM, rd);
        const double sM = exact_quot(left ? -bM : bP, rd);
        // the wave-speed differences, like the face states, must be ordinary numbers
        ok = ok && in_range_pos4(mL + mR, den, mL + mR, den);
        const double w0 = left ? wL[0] : wR[0];
        const double vx = left ? vL - bM : vR - bP;
        const double p = left ? pL : pR;
        const double v = left ? vL : vR;
        const double mf = w0 * vx;
        double f[nh];
        f[0] = mf;
#pragma unroll
        for (int d = 1; d <= NDIM; ++d) {
            f[d] = mf * (left ? wL[d] : wR[d]);
        }
        add_along<NDIM>(f, axis, p);
        f[ie] = (left ? qL[ie] : qR[ie]) * vx + p * v;
#pragma unroll
        for (int i = 0; i < nh; ++i) {
            flux[i] = s_out * f[i];
        }
        add_along<NDIM>(flux, axis, sM * cp);
        flux[ie] += sM * cp * aM;
    } else {
        // flux_from_prim with cons_from_prim's total energy (the same sum)
        double fL[nh], fR[nh];
        const double mfL = wL[0] * vL, mfR = wR[0] * vR;
        fL[0] = mfL;
        fR[0] = mfR;
#pragma unroll
        for (int d = 1; d <= NDIM; ++d) {
            fL[d] = mfL * wL[d];
            fR[d] = mfR * wR[d];
        }
        add_along<NDIM>(fL, axis, pL);
        add_along<NDIM>(fR, axis, pR);
        fL[ie] = (qL[ie] + pL) * vL;
        fR[ie] = (qR[ie] + pR) * vR;
        if constexpr (RS == kRusanov) {
            const double max_c = 0.5 * (csL + fabs(vL) + csR + fabs(vR));
#pragma unroll
            for (int i = 0; i < nh; ++i) {
                flux[i] = 0.5 * (fL[i] + fR[i] - max_c * (qR[i] - qL[i]));
            }
        } else {
            const double sL = smin(-tiny, smin(vL - csL, vR - csR));
            const double sR = smax(-tiny, smax(vL + csL, vL + csR));
            const double den = sR - sL;
            ok = ok && in_range_pos(den);
            const double sM = exact_rcp(den);
#pragma unroll
            for (int i = 0; i < nh; ++i) {
                flux[i] = sM * (sR * fL[i] - sL * fR[i] + sR * sL * (qR[i] - qL[i]));
            }
        }
    }
    return ok;
}

} // namespace mc
