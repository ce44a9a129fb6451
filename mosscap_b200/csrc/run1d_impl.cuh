// The device-driven main loop of a small 1D problem in one launch: a thread-block
// cluster takes a number of whole steps, stages and clock included.
//
// A 1D problem of a thousand cells has about a microsecond of work per stage; launched
// stage by stage, with the clock in between, a step is bound by its launches and by the
// latency of one wave of a few CTAs. Here the state lives in the shared memory of up to
// eight CTAs on neighbouring SMs for the whole launch: the stage buffers are arrays
// distributed over the cluster, a warp takes a 30-cell segment with the stage kernel's
// own sweep (sweep_line), reads its halo from the neighbours' shared memory, and all
// meet at the cluster's hardware barrier after every stage. Ghost cells are not stored:
// a stencil that reaches one reads its source cell and applies the face's transform
// (ghosts stored by the end segments cost these 2600 of 8700 cycles per stage). Each warp
// stores its CFL minimum into every CTA; after the last stage's barrier each thread
// reduces all of them and advances its own copy of the clock, so that every thread takes
// the same dt and the same decision to stop. At the end the state and the last stage's
// input (mc_get_prim) go back to global memory, ghosts included.
//
// run1d_fp64.cu and run1d_fp32.cu define MC_REAL and MC_LAUNCH_NAME and include this.
#pragma once

#include <cuda_runtime.h>

#include "launch.h"
#include "stage_kernels.cuh"

namespace mc {
namespace {

using Real = MC_REAL;

constexpr int kRunCtas = kRun1dCtas;    // CTAs of the cluster at most (portable size)
constexpr int kRunWarps = kRun1dWarps;  // warps of a CTA at most

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// Address of this CTA's shared variable in the CTA of rank `rank`.
__device__ __forceinline__ unsigned remote_addr(const double* addr, unsigned rank) {
    unsigned remote;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(addr)), "r"(rank));
    return remote;
}
__device__ __forceinline__ void store_remote(double* addr, unsigned rank, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote_addr(addr, rank)), "d"(v) : "memory");
}
__device__ __forceinline__ double load_remote(const double* addr, unsigned rank) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote_addr(addr, rank)) : "memory");
    return v;
}

// Interior cell that cell c (interior index, beyond an end of the axis) is a ghost
// of, for a face of kind `kind`: fill_bcs's source (axis_target_at inverted).
__device__ __forceinline__ int ghost_source(int c, int n, int kind) {
    const bool start = c < 0;
    if (kind == kPeriodic) {
        return start ? c + n : c - n;
    }
    if (kind == kZeroGrad || kind == kConstant) {
        return start ? 0 : n - 1;
    }
    return start ? -1 - c : 2 * n - 1 - c;
}

// One stage of segment [x0, x0 + kTile): in, old and out are this CTA's parts of the
// distributed arrays ([var][cells], `cells` cells of each CTA); ghost0, if not null, holds
// the given ghosts of the input ([side][var][ng]).
template <int REC, int LIM, int RS, bool SRC>
__device__ __forceinline__ void run_segment(const StageParams& p, bool last, int combo, int x0, int cells,
                                            unsigned rank, const double* in, const double* old, double* out,
                                            const double* ghost0, Real* W, double dt, double dtdx, Real gfac,
                                            double& dtmin, unsigned& flags) {
    constexpr int NDIM = 1;
    constexpr int nh = 3;
    constexpr int H = halo_of<REC>();
    constexpr int WN = seg1d_window<REC>();
    const int lane = threadIdx.x & 31;
    bool in_range = p.gas.ok != 0;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int it = lane + 32 * u;
        if (it >= WN) {
            continue;
        }
        const int c = x0 - H + it;
        const bool inb = c < p.nx + p.ng;  // H <= ng: the start side never leaves the array
        const bool ghost = c < 0 || c >= p.nx;
        const int side = c < 0 ? 0 : 1;
        double q[kMaxVars];
        if (inb && !(ghost && ghost0)) {
            const int src = ghost ? ghost_source(c, p.nx, p.bc.kind[side]) : c;
            const unsigned owner = (unsigned)src / (unsigned)cells;
            const double* a = in + (src - (int)owner * cells);
#pragma unroll
            for (int v = 0; v < kMaxVars; ++v) {
                q[v] = v < p.nvar ? load_remote(a + v * cells, owner) : 0.0;
            }
            if (ghost) {
                bc_transform<NDIM>(p.bc, 0, side, p.nvar, q);
            }
        } else if (inb) {
#pragma unroll
            for (int v = 0; v < kMaxVars; ++v) {
                q[v] = v < p.nvar ? ghost0[(side * p.nvar + v) * p.ng + (side ? c - p.nx : c + p.ng)] : 0.0;
            }
        } else {
            // outside the array: a benign state that no stored result depends on
#pragma unroll
            for (int v = 0; v < kMaxVars; ++v) {
                q[v] = (v == 0 || v == nh - 1) ? 1.0 : 0.0;
            }
        }
        double w[nh];
        const bool ok = prim_for_sweep<NDIM, Real, vel_low<REC, LIM>()>(p.gamma, p.gas, q, w);
        in_range = in_range && ok;
#pragma unroll
        for (int v = 0; v < nh; ++v) {
            W[v * WN + it] = Real(w[v]);
        }
        if (p.ntracer > 0) {
            const double inv_rho = 1.0 / q[0];
#pragma unroll
            for (int t = 0; t < kMaxVars - nh; ++t) {
                if (t < p.ntracer) {
                    const Real s = Real(q[nh + t] * inv_rho);
                    W[(nh + t) * WN + it] = s;
                    in_range &= sizeof(Real) == 4 || in_range_any<vel_low<REC, LIM>()>(s, s);
                }
            }
        }
        if (inb && !(sizeof(Real) == 8 && ok)) {
            const bool fin = isfinite(q[0]) && isfinite(q[1]) && isfinite(q[2]);
            flags |= state_flags(w[0], w[nh - 1], fin);
        }
    }
    in_range = __all_sync(0xffffffffu, in_range);
    __syncwarp();
    const int cl = lane - 1;  // cell of this lane, relative to x0
    Real d[nh], d_tr[kMaxVars];
    sweep_line<NDIM, REC, LIM, RS, Real>(p, in_range, min(kTile, p.nx - x0), W + H + cl, 1, WN, Real(p.gamma), gfac, 0,
                                         d, d_tr);
    __syncwarp();  // the window is reloaded by the warp's next segment
    const int cell = x0 + cl;
    if (lane >= 1 && lane <= kTile && cell < p.nx) {
        const int o = cell - (int)rank * cells;
        const bool reads_old = combo_reads_old(combo);
        double qi[nh], qo[nh], qu[nh], sdt[nh], qn[kMaxVars];
#pragma unroll
        for (int v = 0; v < nh; ++v) {
            qi[v] = in[v * cells + o];
            qo[v] = reads_old ? old[v * cells + o] : 0.0;
            qu[v] = 0.0;
            qu[v] += double(d[v]);
            qu[v] *= dtdx;
        }
        source_dt_of<NDIM, SRC>(p, qi, dt, sdt);
        combine_all<nh>(combo, qo, qi, qu, sdt, qn);
#pragma unroll
        for (int t = 0; t < kMaxVars - nh; ++t) {
            qn[nh + t] = 0.0;
            if (t < p.ntracer) {
                double qt = 0.0;
                qt += double(d_tr[t]);
                qt *= dtdx;
                const int k = (nh + t) * cells + o;
                qn[nh + t] = combine(combo, reads_old ? old[k] : 0.0, in[k], qt, 0.0);
            }
        }
#pragma unroll
        for (int v = 0; v < kMaxVars; ++v) {
            if (v < p.nvar) {
                out[v * cells + o] = qn[v];
            }
        }
        if (last) {
            dtmin = smin(cfl_bound_of<NDIM, Real>(p, qn, &flags), dtmin);
            // a ghost has its source's bound, but for two kinds of face
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int kind = p.bc.kind[side];
                if ((kind == kDiode || kind == kConstant) && (side ? cell >= p.nx - p.ng : cell < p.ng)) {
                    double g[kMaxVars];
#pragma unroll
                    for (int v = 0; v < kMaxVars; ++v) {
                        g[v] = qn[v];
                    }
                    bc_transform<NDIM>(p.bc, 0, side, p.nvar, g);
                    dtmin = smin(cfl_bound_of<NDIM, Real>(p, g, &flags), dtmin);
                }
            }
        }
    }
}

// Up to `steps` steps from Q; p is a stage's parameters without its buffers, segs the
// segments of a CTA.
template <int REC, int LIM, int RS, bool SRC>
__global__ void __launch_bounds__(kRunWarps * 32)
    run1d_kernel(StageParams p, double* Q, double* last_in, StagePlan plan, int segs, long long steps,
                 double* dt_log) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double mins[kRunCtas * kRunWarps];
    __shared__ double ghost0[2 * kMaxVars * kMaxGhost];
    const unsigned rank = blockIdx.x, ctas = gridDim.x;  // the grid is one cluster
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    const int cells = segs * kTile;
    const int x_first = (int)rank * cells;
    const int own = min(cells, p.nx - x_first);       // not positive in a CTA beyond the last segment
    double* U = reinterpret_cast<double*>(smem_raw);  // [3][nvar][cells]
    const int buf = p.nvar * cells;
    Real* W = reinterpret_cast<Real*>(U + 3 * buf) + (size_t)warp * p.nvar * seg1d_window<REC>();
    for (int k = threadIdx.x; k < cells; k += blockDim.x) {
        for (int v = 0; v < p.nvar; ++v) {
            U[v * cells + k] = k < own ? Q[qidx(p, v, 0, 0, p.ng + x_first + k)] : 0.0;
        }
    }
    for (int k = threadIdx.x; k < 2 * p.nvar * p.ng; k += blockDim.x) {
        const int side = k / (p.nvar * p.ng), r = k - side * p.nvar * p.ng, v = r / p.ng, g = r - v * p.ng;
        ghost0[k] = Q[qidx(p, v, 0, 0, side ? p.ng + p.nx + g : g)];
    }
    DeviceBlock clock = *p.blk;
    const bool log_here = rank == 0 && threadIdx.x == 0;
    const Real gfac = Real((p.gamma + 1.0) / (2.0 * p.gamma));
    bool stepped = false;
    cluster_barrier();
    for (long long k = 0; k < steps && !clock.done; ++k) {
        double dtmin = __longlong_as_double((long long)kInfBits);
        unsigned flags = 0;
        const double dtdx = clock.dt / p.dx;
        for (int st = 0; st < plan.n; ++st) {
            const bool last = st == plan.n - 1;
            for (int j = warp; j < segs; j += warps) {
                const int x0 = x_first + j * kTile;
                if (x0 < p.nx) {
                    run_segment<REC, LIM, RS, SRC>(p, last, plan.combo[st], x0, cells, rank, U + plan.in[st] * buf, U,
                                                   U + plan.out[st] * buf, stepped || st ? nullptr : ghost0, W,
                                                   clock.dt, dtdx, gfac, dtmin, flags);
                }
            }
            if (last) {
                dtmin = warp_min(dtmin);
                if (lane < (int)ctas) {
                    store_remote(&mins[rank * warps + warp], lane, dtmin);
                }
            }
            cluster_barrier();
        }
        stepped = true;
        flags = warp_or(flags);
        if (flags && lane == 0) {
            atomicOr(&p.blk->status, flags);
        }
        double m = __longlong_as_double((long long)kInfBits);
        for (int i = lane; i < (int)ctas * warps; i += 32) {
            m = smin(mins[i], m);
        }
        clock.cfl_min_bits = ordered_bits(warp_min(m));
        clock.status = 0;
        advance_clock(&clock, log_here ? dt_log : nullptr, false, true);
        if (clock.status && log_here) {
            atomicOr(&p.blk->status, clock.status);
        }
    }
    if (stepped) {
        // the state and the last stage's input, each cell with the ghosts it is the
        // source of
        for (int b = 0; b < 2; ++b) {
            StageParams out = p;
            out.q_out = b ? last_in : Q;
            const double* u = U + (b ? plan.in[plan.n - 1] * buf : 0);
            for (int k = threadIdx.x; k < own; k += blockDim.x) {
                double qn[kMaxVars];
#pragma unroll
                for (int v = 0; v < kMaxVars; ++v) {
                    qn[v] = v < p.nvar ? u[v * cells + k] : 0.0;
                }
                unsigned unused = 0;
                write_cell<1, Real>(out, p.ng + x_first + k, 0, 0, qn, false, &unused);
            }
        }
    }
    if (log_here) {
        p.blk->cfl_min_bits = clock.cfl_min_bits;
        p.blk->dt = clock.dt;
        p.blk->time = clock.time;
        p.blk->prev_output_time = clock.prev_output_time;
        p.blk->last_cfl_min = clock.last_cfl_min;
        p.blk->steps = clock.steps;
        p.blk->done = clock.done;
    }
}

struct RunArgs {
    const StageParams& p;
    double* Q;
    double* last_in;
    const StagePlan& plan;
    long long steps;
    double* dt_log;
    cudaStream_t s;
};

template <int REC, int LIM, int RS, bool SRC>
cudaError_t launch_run(const RunArgs& a) {
    const int nseg = (a.p.nx + kTile - 1) / kTile;
    const int ctas = nseg >= kRunCtas ? kRunCtas : nseg >= 4 ? 4 : nseg >= 2 ? 2 : 1;
    const int segs = (nseg + ctas - 1) / ctas;
    const int warps = segs < kRunWarps ? segs : kRunWarps;
    auto k = run1d_kernel<REC, LIM, RS, SRC>;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = sizeof(double) * 3 * (size_t)a.p.nvar * segs * kTile +
                           sizeof(Real) * (size_t)a.p.nvar * warps * seg1d_window<REC>();
    cfg.stream = a.s;
    if (cfg.dynamicSmemBytes > 40 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
        if (e != cudaSuccess) {
            return e;
        }
    }
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ctas;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a.p, a.Q, a.last_in, a.plan, segs, a.steps, a.dt_log);
}

template <int REC, int LIM, int RS>
cudaError_t run_source(const RunArgs& a) {
    return a.p.gravity ? launch_run<REC, LIM, RS, true>(a) : launch_run<REC, LIM, RS, false>(a);
}

template <int REC, int LIM>
cudaError_t run_solver(int rs, const RunArgs& a) {
    return rs == kRusanov ? run_source<REC, LIM, kRusanov>(a)
           : rs == kHll   ? run_source<REC, LIM, kHll>(a)
                          : run_source<REC, LIM, kHllc>(a);
}

template <int REC>
cudaError_t run_limiter(int lim, int rs, const RunArgs& a) {
    return lim == kVanLeer               ? run_solver<REC, kVanLeer>(rs, a)
           : lim == kMonotonizedCentral ? run_solver<REC, kMonotonizedCentral>(rs, a)
                                         : run_solver<REC, kMinmod>(rs, a);
}

} // namespace

cudaError_t MC_LAUNCH_NAME(const StageParams& p, int rec, int lim, int rs, double* Q, double* last_in,
                           const StagePlan& plan, long long steps, double* dt_log, cudaStream_t s) {
    const RunArgs a{p, Q, last_in, plan, steps, dt_log, s};
    switch (rec) {
        case kFog:
            return run_solver<kFog, kMonotonizedCentral>(rs, a);
        case kMuscl:
            return run_limiter<kMuscl>(lim, rs, a);
        case kPpm:
            return run_limiter<kPpm>(lim, rs, a);
        default:
            return run_solver<kWeno5z, kMonotonizedCentral>(rs, a);
    }
}

} // namespace mc
