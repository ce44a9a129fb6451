"""Velocities and mass fractions on both sides of the bounds below which a tile leaves the
branch-free FP64 sweep (2^-800, van Leer slopes 2^-420), down to denormals and zero, against
the C restatement bit for bit: over a uniform medium, where they stay that small through the
stages, and over a random one."""
import numpy as np
import pytest

from mosscap_b200 import problems as P

pytestmark = pytest.mark.gpu

SCHEMES = [("weno5z", "minmod", "hllc"), ("weno5z", "minmod", "hll"), ("weno5z", "minmod", "rusanov"),
           ("ppm", "monotonizedcentral", "hll"), ("ppm", "vanleer", "hllc"), ("ppm", "minmod", "rusanov"),
           ("muscl", "minmod", "hllc"), ("muscl", "monotonizedcentral", "rusanov"), ("muscl", "vanleer", "hll"),
           ("fog", "minmod", "hllc")]
# exponents of the velocities: spread over the range, around either bound, out of it, denormal
SPANS = [(0, 798), (0, 418), (790, 803), (410, 425), (700, 1000), (980, 1080)]


def _state(rng, nd, n, nt, span, uniform, decay):
    shape = (n[2] + 6 if nd > 2 else 1, n[1] + 6 if nd > 1 else 1, n[0] + 6)
    w = np.zeros((2 + nd + nt,) + shape)
    w[0] = 1.3 if uniform else rng.uniform(0.5, 2.0, shape)
    w[1 + nd] = 0.7 if uniform else rng.uniform(0.5, 2.0, shape)
    for v in list(range(1, 1 + nd)) + list(range(2 + nd, 2 + nd + nt)):
        if decay:  # along x, as ahead of a front
            k = -np.linspace(span[0], span[1], shape[2])[None, None, :] + np.zeros(shape)
        else:
            k = -rng.uniform(span[0], span[1], shape)
        # (ldexp of a number in [1, 2): a denormal rounds once)
        x = np.ldexp(rng.uniform(0.2, 0.4, shape), np.floor(k).astype(int)) * rng.choice([-1.0, 1.0], shape)
        w[v] = np.where(rng.random(shape) < 0.1, 0.0, x)
    q = w.copy()
    q[1:1 + nd] *= w[0]
    q[2 + nd:] *= w[0]
    q[1 + nd] = w[1 + nd] / 0.4 + 0.5 * w[0] * (w[1:1 + nd] ** 2).sum(0)
    return q


@pytest.mark.parametrize("span", SPANS)
@pytest.mark.parametrize("nd,n,nt", [(1, (95, 1, 1), 2), (2, (60, 46, 1), 0), (2, (37, 31, 1), 2), (3, (36, 33, 8), 0)])
def test_tiny_velocities_keep_the_reference_bits(gpu_lib, oracle_port, span, nd, n, nt):
    from mosscap_b200.hydro import HydroSim
    for k, (rec, lim, rs) in enumerate(SCHEMES):
        rng = np.random.default_rng(100 * nd + k)
        p = P.Problem("tiny", nd, *n, num_tracers=nt, dx=0.013, reconstruction=rec, slope_limiter=lim,
                      riemann_solver=rs, time_stepper="ssprk3" if k % 2 else "rk2", gamma=1.4, max_cfl=0.2,
                      max_time=1e30, output_delta=1e30,
                      bc=("periodic", "periodic", "wall", "symmetric", "zerograd", "zerograd"))
        for uniform, decay in ((True, False), (True, True), (False, False)):
            p.Q = _state(rng, nd, n, nt, span, uniform, decay)
            sim = HydroSim(p)
            ref = oracle_port.OracleSim(oracle_port.OracleConfig(**p.scheme_fields()), "port")
            ref.set_Q(p.Q)
            sim.fill_bcs()
            ref.fill_bcs()
            dts, rdts = sim.run(2), ref.run(2)
            what = (span, rec, lim, rs, uniform, decay)
            assert np.array_equal(dts.view(np.uint64), rdts.view(np.uint64)), what
            q, r = sim.get_Q() + 0.0, ref.get_Q() + 0.0
            assert np.isfinite(r).all(), what
            bad = np.argwhere(q.view(np.uint64) != r.view(np.uint64))
            assert bad.size == 0, (what, len(bad), bad[:3], [(q[tuple(b)], r[tuple(b)]) for b in bad[:3]])
