// Non-ideal equations of state: the update_eos step that the reference runs
// ahead of every stage's sweep (compute_hydro_fluxes, source/Hydro.cpp:326-
// 328) and once at set-up (source/SetupModules.hpp:253-255). One thread per
// cell, ghosts included, as the reference's FlatLoop over zc x yc x xc.
//
//  * analytic LTE hydrogen (source/AnalyticLteH.hpp:49-120): temperature and
//    ionisation fraction of every cell by bisection on the Saha equation;
//    the state is not changed.
//  * tabulated LTE hydrogen (source/TabulatedLteH.hpp:60-163): y and
//    log10 T by bilinear interpolation in (log10(eint / rho), log10 rho),
//    and the energy shifted by the ionisation energy of the change of y
//    since the previous call.
//
// Compiled without contraction and with the reference's expression trees;
// pow, exp and log10 are CUDA's, whose last bits can differ from the C
// library's, so results agree with the reference to rounding, not bit for
// bit. A condition on which the reference aborts (bisection bounds flipped,
// negative internal energy) raises MC_FLAG_EOS in the status instead; the
// tabulated kind leaves such a cell (and any cell whose table coordinates
// are not numbers) unchanged.
#include <cuda_runtime.h>

#include "common.cuh"
#include "eos.h"

namespace mc {
namespace {

constexpr double kHMass = 1.6737830080950003e-27;  // [kg]
constexpr double kKB = 1.380649e-23;               // [J / K]
constexpr double kChiH = 2.178710282685096e-18;    // [J]

// IEEE division and the ionisation fraction with it, for operands outside exact_fp64.cuh's.
__device__ __noinline__ double div_any(double a, double b) {
    return a / b;
}
__device__ __noinline__ double y_any(double nhtot, double X) {
    return 0.5 * (-X + sqrt(X * X + 4 * nhtot * X)) / nhtot;
}

// Positive and in [2^-400, 2^340).
__device__ __forceinline__ bool lte_range(double x) {
    return (unsigned)(__double2hiint(x) - 0x26f00000) < 0x55300000u - 0x26f00000u;
}

// One cell's F(T) = T - T(y(T)) and its y (source/AnalyticLteH.hpp:49-76). With !PLAIN the
// quotients and the root are exact_fp64.cuh's, for operands that meet its conditions: X,
// e_to_T and T in lte_range and n in it above 2^-40. Then -X + sqrt(X^2 + 4 n X) is zero or
// at least an ulp of X, 2^-452, and y, rounding errors of that included, below 2^330. The
// same bits.
template <bool PLAIN>
struct LteCell {
    double nhtot, e_to_T, eint, rho, inv_avg_mass;
    double ion_e;  // 1 with the ionisation energy, 0 without
    Recip rn;
    bool n_ok, e_ok;
    __device__ __forceinline__ LteCell(double rho_, double nhtot_, double e_to_T_, double eint_, double ion_e_,
                                       double inv_avg_mass_) {
        rho = rho_;
        nhtot = nhtot_;
        e_to_T = e_to_T_;
        eint = eint_;
        ion_e = ion_e_;
        inv_avg_mass = inv_avg_mass_;
        n_ok = !PLAIN && lte_range(nhtot) && nhtot >= 0x1p-40;
        e_ok = !PLAIN && lte_range(e_to_T);
        rn = recip_of(nhtot);
    }
    // small: y is below 2^330
    __device__ __forceinline__ double temp_from_y(double y, bool small) const {
        const double d = 1.0 + y;
        const double t = e_ok && small ? exact_div(e_to_T, d) : PLAIN ? e_to_T / d : div_any(e_to_T, d);
        return t * (eint - ion_e * y * rho * (kChiH / kHMass) * inv_avg_mass);
    }
    __device__ __forceinline__ double f_of(double temp, double& y) const {
        bool small;
        y = y_of(temp, small);
        return temp - temp_from_y(y, small);
    }
    __device__ __forceinline__ double y_of(double temp, bool& small) const {
        const double chi = -157763.42386247337;
        const double a = !PLAIN && lte_range(temp) ? exact_div(chi, temp) : PLAIN ? chi / temp : div_any(chi, temp);
        const double X = 2.4146830395719654e+21 * pow(temp, 1.5) * exp(a);
        small = n_ok && lte_range(X);
        if (small) {
            return exact_quot(0.5 * (-X + exact_sqrt(X * X + 4 * nhtot * X)), rn);
        }
        return PLAIN ? 0.5 * (-X + sqrt(X * X + 4 * nhtot * X)) / nhtot : y_any(nhtot, X);
    }
};

template <int NDIM>
__device__ __forceinline__ void energies(const double* q, long long id, long long plane, double& rho, double& e_kin,
                                         double& eint) {
    double mom2_sum = q[id + plane] * q[id + plane];
    if constexpr (NDIM > 1) {
        mom2_sum += q[id + 2 * plane] * q[id + 2 * plane];
    }
    if constexpr (NDIM > 2) {
        mom2_sum += q[id + 3 * plane] * q[id + 3 * plane];
    }
    rho = q[id];
    e_kin = 0.5 * mom2_sum / rho;
    eint = q[id + (1 + NDIM) * plane] - e_kin;
}

// The temperature at which the energy of a cell and its ionisation agree, in FP32 and
// to FP32's accuracy: the root in [t0, t1] of F(T) = T - t1 (1 - k y) / (1 + y) with
// y^2 / (1 - y) = c T^1.5 exp(-157763.4 / T), by Newton steps kept inside the bracket;
// slope: F' there.
__device__ __forceinline__ float lte_root_estimate(float t0, float t1, float c, float k, float& slope) {
    float lo = t0, hi = t1, t = 0.5f * (t0 + t1);
    for (int it = 0; it < 16; ++it) {
        const float it_ = __fdividef(1.0f, t);
        const float r = c * t * __fsqrt_rn(t) * __expf(-157763.42f * it_);
        const float y = __fdividef(2.0f, 1.0f + __fsqrt_rn(1.0f + __fdividef(4.0f, r)));
        const float w = __fdividef(1.0f, 1.0f + y);
        const float f = t - t1 * (1.0f - k * y) * w;
        const float dy = y * (1.0f - y) * __fdividef(1.5f * it_ + 157763.42f * it_ * it_, 2.0f - y);
        const float df = 1.0f + t1 * dy * w * ((1.0f - k * y) * w + k);
        if (f > 0.0f) {
            hi = t;
        } else {
            lo = t;
        }
        slope = df;
        const float n = t - __fdividef(f, df);
        const float before = t;
        t = (n >= lo && n <= hi) ? n : 0.5f * (lo + hi);
        if (fabsf(t - before) < 1e-6f * t) {
            break;
        }
    }
    return t;
}

// A cell's F and how far its evaluation in FP64 can be off, all in FP32: amp = t1 (1 + k) and
// c of lte_root_estimate. The evaluation's error at T is at most
// u t1 (1 + k) ((r + 2) / (1 + y)^2 + 5 + (10 + 157763.4 / T) y (1 - y) / ((2 - y) (1 + y)^2)),
// u = 2^-53, r = X / n = c T^1.5 exp(-157763.4 / T): dT/dy = -t1 (1 + k) / (1 + y)^2 times
// y's error, which is that of -X + sqrt(X^2 + 4 n X) (sqrt's argument off by 2 u, its own
// rounding u: u (X + 2 n) / n) and that of X itself (pow, exp and its argument), and
// temp_from_y's own roundings. With 1 + y >= (1 + 2 r) / (1 + r), T >= 100 and the last
// fraction at most 0.08 it is below u amp (r / 4 + 160), which grows with T.
constexpr float kLteErrorMax = 0.0045f;  // [K]; twice this is below the replay's margin of 0.01
struct LteError {
    float amp, c;
    __device__ __forceinline__ float operator()(float T) const {
        const float r = c * (T * T) * rsqrtf(T) * __expf(__fdividef(-157763.42f, T));
        return 1.1103e-16f * amp * (0.25f * r + 160.0f);
    }
    // Whether the error stays within the limit from `hi` up to where F is large, for tests up to t1.
    __device__ __forceinline__ bool allows(float hi, float t1) const {
        return (*this)(fminf(hi + 1.0f + (*this)(t1), t1)) < kLteErrorMax;
    }
};

// The reference's bisection (source/AnalyticLteH.hpp:78-119) halves [T(y = 1), T(y = 0)]
// about 17 times, with a pow, an exp and a root for each test temperature: FP64-bound. Its
// outcome is fixed by the signs of F(T) = T - T(y(T)) at the test temperatures and by
// whether |F| < 0.1 there. F' >= 1 (y grows with T, and T(y) falls with y), so one value
// F(r) bounds the root: it lies between r and r - F(r); and a test temperature more than
// 0.1 beyond that bracket has a known sign and |F| > 0.1. So the bisection is replayed, and
// F evaluated, with the same expressions, only at an FP32 estimate of the root, at the test
// temperatures near it and at the last one (whose y is the result): 2.3 evaluations per cell
// where it took 15 (1e-9 .. 1e-6 kg/m^3, 5e3 .. 2e4 K; 3.3 and 18 with the ionisation energy).
// Both values are evaluated with an error: 0.11 in place of 0.1 leaves 0.01 for that of the
// bracket's and that of the skipped one together. Each bracketing evaluation is at a
// temperature where the error is at most kLteErrorMax, and it must stay so up to hi + 1 +
// its largest value, beyond which F exceeds it by more than 0.1 in any case. Cells that
// do not meet this, and those outside the argument (non-positive or non-finite density or
// energy, flipped bounds), are evaluated at every step.
// PLAIN: every cell is (the same bits; for comparison).
// One update of 512^2 smooth cells (B200), IEEE divisions and every step evaluated -> this
// kernel: 68 -> 33 us around 1e4 K and 3e-8 kg/m^3, 83 -> 75 with the ionisation energy; 62 ->
// 27 and 64 -> 28 around 5e3 K and 1e-4; where F is mostly rounding error and no bracket is
// allowed 101 -> 97 and 101 -> 97 (1e6 K, 1e-12), 78 -> 76 and 85 -> 86 (4e4 K, 1e-10), 83 -> 82
// and 87 -> 87 (1e5 K, 1e-8). Four CTAs per SM: the registers of three take 91 us in the second.
template <int NDIM, bool PLAIN = false>
__global__ void __launch_bounds__(256, 4) eos_analytic_kernel(EosLaunch L) {
    if (L.blk && L.skip_when_done && L.blk->done) {
        return;
    }
    const double gamma = L.gamma;
    const double ionisation_e = L.ionisation_e ? 1.0 : 0.0;
    const double inv_avg_mass = 1.0 / L.avg_mass;
    // t1 k of lte_root_estimate: the same for every cell
    const float t1k = L.ionisation_e ? (float)(kChiH / kKB * (gamma - 1.0)) : 0.0f;
    unsigned flags = 0;
    for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < L.plane;
         id += (long long)gridDim.x * blockDim.x) {
        double rho, e_kin, eint;
        energies<NDIM>(L.q_in, id, L.plane, rho, e_kin, eint);
        const double e_to_T = (gamma - 1.0) / (rho * (kKB / kHMass) * inv_avg_mass);
        const double nhtot = rho * ((1.0 / kHMass) * inv_avg_mass);
        const LteCell<PLAIN> cell(rho, nhtot, e_to_T, eint, ionisation_e, inv_avg_mass);
        const double min_temperature = 100.0;
        const double t1 = cell.temp_from_y(1.0, true);
        const double tb0 = (t1 < min_temperature) ? min_temperature : t1;  // std::max
        const double tb1 = cell.temp_from_y(0.0, true);
        if (tb0 > tb1) {
            flags |= kFlagEos;
        }
        double temp_step = tb1 - tb0;
        double temp = tb0;
        double y = 0.0;
        // the root's bracket; (-inf, inf): every test temperature is evaluated
        double lo = -__longlong_as_double(0x7ff0000000000000ll), hi = -lo;
        double test_temp = 0.0;
        LteError error{0.0f, 0.0f};
        float slope = 1.0f;
        bool bracket = false;
        int iter = 0;  // tests so far; negative: evaluations for the bracket
        const float nf = (float)nhtot, t0f = (float)tb0, t1f = (float)tb1;
        // (density and, tb0 being at least 100, energy are positive)
        if (!PLAIN && gamma > 1.0 && nf > 0.0f && t1f > t0f) {
            error.amp = t1f + t1k;
            error.c = __fdividef(2.4146830e21f, nf);
            if (error(t0f) < kLteErrorMax) {
                const float root = lte_root_estimate(t0f, t1f, error.c, __fdividef(t1k, t1f), slope);
                if (error(root) < kLteErrorMax && error.allows(root, t1f)) {
                    test_temp = (double)root;
                    bracket = true;
                    iter = -2;
                }
            }
        }
        if (PLAIN || !__any_sync(__activemask(), bracket)) {
            // no lane has a bracket: the plain loop
            for (iter = 0; iter < 100; ++iter) {
                temp_step *= 0.5;
                test_temp = temp + temp_step;
                const double temp_err = cell.f_of(test_temp, y);
                if (temp_err <= 0.0) {
                    temp = test_temp;
                }
                if (fabs(temp_step) < 1e-1 || fabs(temp_err) < 1e-1) {
                    break;
                }
            }
            iter = 100;
        }
        while (iter < 100) {
            // tests whose outcome the bracket decides; a test with the last
            // y of the cell (the step below 0.1, or the 100th) is evaluated
            if (iter >= 0) {
                for (;;) {
                    temp_step *= 0.5;
                    test_temp = temp + temp_step;
                    ++iter;
                    const bool above = test_temp - 0.11 > hi;
                    const bool below = test_temp + 0.11 < lo;
                    if (!(above || below) || fabs(temp_step) < 1e-1 || iter == 100) {
                        break;
                    }
                    if (below) {
                        temp = test_temp;
                    }
                }
            }
            double yt;
            const double temp_err = cell.f_of(test_temp, yt);
            if (bracket && temp_err > 0.0) {
                hi = test_temp < hi ? test_temp : hi;
                lo = test_temp - temp_err > lo ? test_temp - temp_err : lo;
            } else if (bracket && temp_err <= 0.0) {
                lo = test_temp > lo ? test_temp : lo;
                hi = test_temp - temp_err < hi ? test_temp - temp_err : hi;
            }
            if (iter < 0) {
                // a steep F leaves a wide bracket: once more, somewhat beyond the
                // Newton step from here, where F mostly has the other sign
                const double next = test_temp - 1.5 * temp_err / (double)slope;
                if (iter == -2 && fabs(temp_err) > 0.1 && error((float)next) < kLteErrorMax) {
                    iter = -1;
                    test_temp = next;
                    continue;
                }
                iter = 0;
                if (!error.allows((float)hi, t1f)) {
                    bracket = false;
                    hi = __longlong_as_double(0x7ff0000000000000ll);
                    lo = -hi;
                }
                continue;
            }
            y = yt;
            if (temp_err <= 0.0) {
                temp = test_temp;
            }
            if (fabs(temp_step) < 1e-1 || fabs(temp_err) < 1e-1) {
                break;
            }
        }
        L.y[id] = y;
        L.T[id] = temp;
    }
    if (flags && L.blk) {
        atomicOr(&L.blk->status, flags);
    }
}

struct Sample {
    double y, log_T;
};

__device__ __forceinline__ Sample table_sample(const EosLaunch& L, const double* Y, const double* LT,
                                              double log_eint_rho, double log_rho) {
    const double frac_eint_rho = (log_eint_rho - L.x_start) / L.x_step;
    int ix = int(floor(frac_eint_rho));
    int ixp;
    double tx, txp;
    const int max_x = L.nx_tab - 1;
    const int max_y = L.ny_tab - 1;
    if (frac_eint_rho < 0.0 || frac_eint_rho >= max_x) {
        ix = ix < 0 ? 0 : ix;
        ix = max_x < ix ? max_x : ix;
        ixp = ix;
        tx = 1.0;
        txp = 0.0;
    } else {
        ixp = ix + 1;
        txp = frac_eint_rho - ix;
        tx = 1.0 - txp;
    }
    const double frac_rho = (log_rho - L.y_start) / L.y_step;
    int iy = int(floor(frac_rho));
    int iyp;
    double ty, typ;
    if (frac_rho < 0.0 || frac_rho >= max_y) {
        iy = iy < 0 ? 0 : iy;
        iy = max_y < iy ? max_y : iy;
        iyp = iy;
        ty = 1.0;
        typ = 0.0;
    } else {
        iyp = iy + 1;
        typ = frac_rho - iy;
        ty = 1.0 - typ;
    }
    const int n = L.nx_tab;
    Sample s;
    s.y = (ty * (tx * Y[iy * n + ix] + txp * Y[iy * n + ixp]) + typ * (tx * Y[iyp * n + ix] + txp * Y[iyp * n + ixp]));
    s.log_T = (ty * (tx * LT[iy * n + ix] + txp * LT[iy * n + ixp]) +
               typ * (tx * LT[iyp * n + ix] + txp * LT[iyp * n + ixp]));
    return s;
}

// With tables_in_smem, a persistent grid whose CTAs first copy both tables
// into shared memory: each cell then gathers its eight table values from
// shared memory instead of waiting on global loads after its state loads.
template <int NDIM>
__global__ void __launch_bounds__(256) eos_tabulated_kernel(EosLaunch L, int tables_in_smem) {
    if (L.blk && L.skip_when_done && L.blk->done) {
        return;
    }
    extern __shared__ __align__(16) double tab_smem[];
    const double* Y = L.y_table;
    const double* LT = L.log_T_table;
    if (tables_in_smem) {
        const int n = L.nx_tab * L.ny_tab;
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            tab_smem[k] = L.y_table[k];
            tab_smem[n + k] = L.log_T_table[k];
        }
        __syncthreads();
        Y = tab_smem;
        LT = tab_smem + n;
    }
    constexpr int ie = 1 + NDIM;
    constexpr int nh = 2 + NDIM;
    constexpr int U = 4;  // cells per thread whose loads are issued together
    const long long stride = (long long)gridDim.x * blockDim.x;
    unsigned flags = 0;
    for (long long base = blockIdx.x * (long long)blockDim.x + threadIdx.x; base < L.plane; base += U * stride) {
        double qv[U][nh], yp[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long id = base + u * stride;
            if (id < L.plane) {
#pragma unroll
                for (int v = 0; v < nh; ++v) {
                    qv[u][v] = L.q_in[id + v * L.plane];
                }
                yp[u] = L.y[id];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long id = base + u * stride;
            if (id >= L.plane) {
                continue;
            }
            const double* q = qv[u];
            double mom2_sum = q[1] * q[1];
            if constexpr (NDIM > 1) {
                mom2_sum += q[2] * q[2];
            }
            if constexpr (NDIM > 2) {
                mom2_sum += q[3] * q[3];
            }
            const double rho = q[0];
            const double e_kin = 0.5 * mom2_sum / rho;
            const double eint = q[ie] - e_kin;
            const double log_rho = log10(rho);
            const double log_eint_rho = log10(eint) - log_rho;
            // The reference aborts on eint < 0 (TabulatedLteH.hpp:142-144); a
            // NaN coordinate (eint < 0, rho <= 0 or a non-finite state) would
            // also index the table out of range. Flag the cell and leave it.
            const double fx = (log_eint_rho - L.x_start) / L.x_step;
            const double fy = (log_rho - L.y_start) / L.y_step;
            if (eint < 0.0 || fx != fx || fy != fy) {
                flags |= kFlagEos;
                continue;
            }
            const Sample s = table_sample(L, Y, LT, log_eint_rho, log_rho);
            const double prev_y = yp[u];
            L.y[id] = s.y;
            const double delta_eint = (prev_y < 0.0) ? 0.0 : rho * (kChiH / kHMass) * (s.y - prev_y);
            L.T[id] = pow(10.0, s.log_T);
            // the state with the energy shifted: in place, or into a copy when
            // the input must stay as it is (the step-start state)
            if (L.q_out != L.q_in) {
                for (int v = 0; v < L.nvar; ++v) {
                    if (v != ie) {
                        L.q_out[id + v * L.plane] = L.q_in[id + v * L.plane];
                    }
                }
            }
            L.q_out[id + ie * L.plane] = q[ie] + delta_eint;
        }
    }
    if (flags && L.blk) {
        atomicOr(&L.blk->status, flags);
    }
}

constexpr size_t kTableSmemMax = 74 * 1024;  // three CTAs per SM (228 KB)

template <class K>
cudaError_t allow_table_smem(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) {
        return cudaSuccess;
    }
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

} // namespace

cudaError_t launch_eos_analytic_plain(const EosLaunch& L, cudaStream_t s) {
    const long long want = (L.plane + 255) / 256;
    eos_analytic_kernel<1, true><<<(int)(want < 148 * 16 ? want : 148 * 16), 256, 0, s>>>(L);
    return cudaGetLastError();
}

cudaError_t launch_eos_update(const EosLaunch& L, int ndim, cudaStream_t s) {
    const long long want = (L.plane + 255) / 256;
    const int blocks = (int)(want < 148 * 16 ? want : 148 * 16);
    if (L.type == kEosAnalytic) {
        if (ndim == 1) {
            eos_analytic_kernel<1><<<blocks, 256, 0, s>>>(L);
        } else if (ndim == 2) {
            eos_analytic_kernel<2><<<blocks, 256, 0, s>>>(L);
        } else {
            eos_analytic_kernel<3><<<blocks, 256, 0, s>>>(L);
        }
    } else if (L.type == kEosTabulated) {
        // both tables in shared memory when they fit three CTAs per SM
        const size_t tab_bytes = 2 * sizeof(double) * (size_t)L.nx_tab * (size_t)L.ny_tab;
        const bool smem = tab_bytes <= kTableSmemMax;
        const size_t sm = smem ? tab_bytes : 0;
        const int grid = smem ? (int)(want < 148 * 3 ? want : 148 * 3) : blocks;
        cudaError_t e = cudaSuccess;
        if (ndim == 1) {
            e = allow_table_smem(eos_tabulated_kernel<1>, sm);
            eos_tabulated_kernel<1><<<grid, 256, sm, s>>>(L, smem ? 1 : 0);
        } else if (ndim == 2) {
            e = allow_table_smem(eos_tabulated_kernel<2>, sm);
            eos_tabulated_kernel<2><<<grid, 256, sm, s>>>(L, smem ? 1 : 0);
        } else {
            e = allow_table_smem(eos_tabulated_kernel<3>, sm);
            eos_tabulated_kernel<3><<<grid, 256, sm, s>>>(L, smem ? 1 : 0);
        }
        if (e != cudaSuccess) {
            return e;
        }
    }
    return cudaGetLastError();
}

} // namespace mc
