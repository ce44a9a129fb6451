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
// quotient: 7 FP64 instructions per quotient, 5 for a further quotient with
// the same denominator, 8 per root, all of them free to overlap.
//
// Where a product with a power of two feeds an addition the two are written
// as one fma: the product is exact, so the result is the same rounding of the
// same sum as in physics.cuh. Everything else keeps the order of
// physics.cuh, whose functions are evaluated instead (generic form) wherever
// a range test fails.
//
// What an FP64 instruction costs (measured, 20 warps per SM): two cycles of an SM
// sub-partition for products, sums and fmas that read at most two distinct registers
// (a constant or a repeated operand as the third), three for an fma of three
// registers. So the refinements prefer the forms 1 - b y, e + e e and t + t s.
// With the sweeps' code as it is these cycles are what bounds them (2D WENO5-Z).
//
// Division. With the seed y = (1/b)(1 - e) and s = e + e^2, (1/b) = y (1 + s) up to a
// factor 1 + e^3. q = t + t s with t = a y is within 1.02 ulp of a/b (t's
// rounding, its own, e^3 <= 2^-59.8), the residual d = b q - a is exact, and the
// result q - (d + d s) y is a/b rounded once, but for an error of c = d / b of
// relatively 2^-53 / m + 2^-59.8, m in [1, 2) the significand of d + d s, b's up to
// 2^-19.9. That can only matter for a/b near a rounding boundary, where |c| is half an ulp.
// With 53-bit integers A, B as the operands' significands a quotient is at least
// 1 / (2B) ulp away from a boundary (it cannot lie on one), that is 2^-53 / b ulp,
// and the error is (2^-54 / b) (1 + 2^-5.8) ulp: about half of it. (Markstein, IBM J.
// Res. Dev. 34, 1990, has the correction by an exact residual, and this way of
// bounding it.) Two things need a closer look. For b within 2^-26 of 2, B = 2^53 - k, the
// seed is 1/2 exactly and d + d s can pass the next power of two, where m is 1: for
// the closest quotient it lies k 2^-54 units above the middle between two doubles, and
// the rounding of s moves it by less than that unless k = 1, where by as much; s is
// therefore rounded up, which settles 1 / (2 - 2^-52). And for q a power of two and
// a/b below it, where an ulp is half as long, a boundary is also at three quarters of q's
// ulp (the one at a quarter is out of reach, a/b = 1 - n/B with integer n): n = 1 and B
// next to 2^54 / 3, two quotients. Both kinds are tested with the closest quotients of
// many other B (tests/test_exact_ops_gpu.py).
//
// The seed rcp.approx.ftz.f64 has a relative error <= 2^-19.93 over all of its
// inputs (it reads the operand's upper word only; measured over all of them).
//
// Square root (Cornea-Hasegan, Golliver and Markstein, ARITH-14, 1999, for the
// form and the enumeration of the hard cases): seed rsqrt.approx.ftz.f64
// (<= 2^-20.0), one third-order step for root and half reciprocal, one exact
// residual. The value before the last rounding is within 2^-102.8 of the root of
// x in [1, 4); a root at odd distance j from a rounding boundary, in units where
// the boundary's square is an integer, is at least j 2^-108 from it, so only
// j <= 37 can round differently; all significands with j < 256 are tested.
//
// Measured (B200, KH 2048^2 WENO5-Z + HLLC, one stage, bit-identical): IEEE division and
// root 0.594 ms; quotients by two Newton steps and two corrections (nine instructions)
// 0.506 ms; this form 0.453 ms. Six instructions without d s, a test of d against
// half an ulp (four integer instructions) and the lines where it fires
// evaluated again: 0.514 ms, the test alone 0.038 ms.
#pragma once

#include <cmath>

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

// A denominator: y = (1/b)(1 - e), s = e + e^2.
struct Recip {
    double b, y, s;
};
__device__ __forceinline__ Recip recip_of(double b) {
    Recip r;
    r.b = b;
    r.y = rcp_seed(b);
    const double e = fma(-b, r.y, 1.0);
    r.s = __fma_ru(e, e, e);
    return r;
}

// RN(a / b) for b whose reciprocal is normal and a that is zero (the result is a
// zero of either sign: no result of the stage kernels depends on it) or so
// that the quotient is normal and |a| > 2^-960 (the residual's last bit, 2^-106 of a, is
// then a double).
__device__ __forceinline__ double exact_quot(double a, const Recip& r) {
    const double t = __dmul_rn(a, r.y);
    const double q = fma(t, r.s, t);
    double d = fma(r.b, q, -a);
    d = fma(d, r.s, d);
    return fma(-d, r.y, q);
}
__device__ __forceinline__ double exact_div(double a, double b) {
    return exact_quot(a, recip_of(b));
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
// and mass fraction is zero or of magnitude in [2^-800, 2^100) ([2^-420, 2^100) where
// a van Leer slope multiplies two of their differences). Then every division and root
// below meets its conditions or its result does not matter:
//   a momentum that is not zero is at least 2^-920, and differences of such velocities
//   are zero or at least an operand's last bit, 2^-852 (2^-472: their products 2^-944);
//   factors 2 and fmas in place of products with a power of two are exact at these sizes;
//   WENO5-Z: squares of differences below 2^-537 vanish, as in physics.cuh, beside the
//   regulariser 2^-119.6; the weights are at least 1 and at most 2^650; the weighted sum is
//   zero or at least 2^-904, and its quotient by the weights' sum normal: where a weight is
//   large, its own term of the sum, or, where that is zero, a large cell's, is too;
//   kinetic energies, momentum fluxes and wave-speed terms of velocities this small are
//   formed by the same operations as in physics.cuh, or vanish beside p >= 2^-120.
// The face states a reconstruction makes of them are tested again before the Riemann solver
// (positivity is not kept by it). Upper words as integers: one or two instructions of
// the integer pipe for each value, none of the FP64 pipe.
// Velocities decay to nothing ahead of a front in a uniform medium, so their bound is as low
// as this allows: KH 2048^2 with the velocities across the flow times 1e-200, WENO5-Z, 2.64
// -> 1.38 ms per step against a bound of 2^-250. Denormal ones stay out: Sedov 256^3 has
// them in 5 to 7 % of its tiles from step 20 on and takes 7.42 ms per step at step 10, 7.56 at
// 20, 7.59 at 40 and 7.65 at 80 (10.15 throughout with IEEE divisions).
constexpr unsigned kVelLow = 0x0df00000u;         // upper word of 2^-800
constexpr unsigned kVelLowVanLeer = 0x25b00000u;  // 2^-420
template <int REC, int LIM>
__host__ __device__ constexpr unsigned vel_low() {
    return LIM == kVanLeer && (REC == kMuscl || REC == kPpm) ? kVelLowVanLeer : kVelLow;
}
__device__ __forceinline__ bool in_range_pos(double x) {
    return (unsigned)(__double2hiint(x) - 0x38700000) < 0x46300000u - 0x38700000u;
}
template <unsigned LOW>
__device__ __forceinline__ bool in_range_magnitude(double x) {
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) - LOW < 0x46300000u - LOW;
}
// x, a quotient with numerator n.
template <unsigned LOW>
__device__ __forceinline__ bool in_range_any(double x, double n) {
    // (no branch: the loads of the next values do not wait)
    return in_range_magnitude<LOW>(x) |
           ((((unsigned)__double2hiint(n) & 0x7fffffffu) | (unsigned)__double2loint(n)) == 0u);
}
// Four upper words of positive values at once.
__device__ __forceinline__ bool in_range_pos4(double a, double b, double c, double d) {
    const int ha = __double2hiint(a), hb = __double2hiint(b), hc = __double2hiint(c), hd = __double2hiint(d);
    return min(min(ha, hb), min(hc, hd)) >= 0x38700000 && max(max(ha, hb), max(hc, hd)) < 0x46300000;
}

// The constants of the gas of one launch, formed on the host (kernel
// parameters: constant-bank operands, no registers).
struct FastGas {
    double gm1, gfac;    // gamma - 1, (gamma + 1) / (2 gamma)
    double rgm1, sgm1;   // RN(1 / (gamma - 1)) and its residual (Recip's y and s)
    int ok;              // gamma and gamma - 1 in [2^-20, 2^20]
};
inline FastGas fast_gas(double gamma) {
    FastGas g;
    g.gm1 = gamma - 1.0;
    g.gfac = (gamma + 1.0) / (2.0 * gamma);
    g.rgm1 = 1.0 / g.gm1;
    g.sgm1 = std::fma(-g.gm1, g.rgm1, 1.0);
    g.ok = gamma <= 0x1p20 && g.gm1 >= 0x1p-20 ? 1 : 0;
    return g;
}

// ---- physics.cuh's functions for values in range -------------------------------

// prim_from_cons; false: the cell is out of range and w holds no result.
template <int NDIM, unsigned LOW>
__device__ __forceinline__ bool fast_prim(double gm1, const double* q, double* w) {
    const Recip r = recip_of(q[0]);
    w[0] = q[0];
#pragma unroll
    for (int d = 1; d <= NDIM; ++d) {
        w[d] = exact_quot(q[d], r);
    }
    bool ok = true;
    double v2 = 0.0;
#pragma unroll
    for (int d = 1; d <= NDIM; ++d) {
        ok = ok && in_range_magnitude<LOW>(w[d]);
        v2 = d == 1 ? __dmul_rn(w[d], w[d]) : __dadd_rn(v2, __dmul_rn(w[d], w[d]));
    }
    // E - (0.5 rho) v2: the factor 1/2 is exact
    w[1 + NDIM] = __dmul_rn(gm1, fma(-0.5, __dmul_rn(q[0], v2), q[1 + NDIM]));
    if (!ok) {
        // velocities that are zero, by their momenta (a quotient may vanish beside a momentum
        // that does not; tested here and not for every cell: KH 2048^2 step -0.4 %)
        ok = true;
#pragma unroll
        for (int d = 1; d <= NDIM; ++d) {
            ok = ok && in_range_any<LOW>(w[d], q[d]);
        }
    }
    return ok && in_range_pos(q[0]) && in_range_pos(w[1 + NDIM]);
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
    // v2 below 2^-900 leaves cs + |v| = cs
    const double vel = __double2hiint(v2) < 0x07b00000 ? 0.0 : exact_sqrt(v2);
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
    const Recip rg{gas.gm1, gas.rgm1, gas.sgm1};
    // total energy of a state (0.5 rho v^2 with an exact 1/2)
    auto energy = [&](const double* w) {
        double k = w[1] * w[1];
#pragma unroll
        for (int d = 2; d <= NDIM; ++d) {
            k += w[d] * w[d];
        }
        return fma(0.5, w[0] * k, exact_quot(w[ie], rg));
    };
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
        const double vxL = vL - aL;
        const double vxR = vR - aR;
        const double tL = pL + vxL * (wL[0] * vL);
        const double tR = pR + vxR * (wR[0] * vR);
        const double mL = wL[0] * vxL;
        const double mR = -(wR[0] * vxR);
        const Recip rm = recip_of(mL + mR);
        const double aM = exact_quot(tL - tR, rm);
        const double cp = smax(exact_quot(mL * tR + mR * tL, rm), 0.0);
        const bool left = aM >= 0.0;
        const double den = left ? (aM - bM) : (bP - aM);
        const Recip rd = recip_of(den);
        const double s_out = exact_quot(left ? aM : -aM, rd);
        const double sM = exact_quot(left ? -bM : bP, rd);
        // the wave-speed differences, like the face states, must be ordinary numbers
        ok = ok && in_range_pos(rm.b) && in_range_pos(den);
        // the upwind side only: the other's flux has weight zero. For finite g
        // s f + 0 g is s f, but for the sign of a zero, and no result depends on
        // that: every flux difference is added to a sum that starts from +0
        double w[nh];
#pragma unroll
        for (int i = 0; i < nh; ++i) {
            w[i] = left ? wL[i] : wR[i];
        }
        const double v = left ? vL : vR;
        const double vx = v - (left ? bM : bP);
        const double mf = w[0] * vx;
        double f[nh];
        f[0] = mf;
#pragma unroll
        for (int d = 1; d <= NDIM; ++d) {
            f[d] = mf * w[d];
        }
        add_along<NDIM>(f, axis, w[ie]);
        f[ie] = energy(w) * vx + w[ie] * v;
#pragma unroll
        for (int i = 0; i < nh; ++i) {
            flux[i] = s_out * f[i];
        }
        add_along<NDIM>(flux, axis, sM * cp);
        flux[ie] += sM * cp * aM;
    } else {
        // momenta and energies; flux_from_prim's total energy is the same sum
        double qL[nh], qR[nh], fL[nh], fR[nh];
        qL[0] = wL[0];
        qR[0] = wR[0];
#pragma unroll
        for (int d = 1; d <= NDIM; ++d) {
            qL[d] = wL[0] * wL[d];
            qR[d] = wR[0] * wR[d];
        }
        qL[ie] = energy(wL);
        qR[ie] = energy(wR);
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
            const double sM = exact_div(1.0, den);
#pragma unroll
            for (int i = 0; i < nh; ++i) {
                flux[i] = sM * (sR * fL[i] - sL * fR[i] + sR * sL * (qR[i] - qL[i]));
            }
        }
    }
    return ok;
}

} // namespace mc
