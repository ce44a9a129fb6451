"""The one-launch main loop of small 1D problems (csrc/run1d_impl.cuh): against the C
restatement and, in the FP32 form, against the loop of separate launches (which a
CFL-reduction hook asks for), bit for bit. Sizes around one segment, one CTA, the
cluster's warps, its largest problem and the first one beyond it."""
import numpy as np
import pytest

from mosscap_b200 import problems as P

pytestmark = pytest.mark.gpu

BCS = [("zerograd",) * 6, ("periodic",) * 6, ("wall", "symmetricoutflowdiode") + ("zerograd",) * 4,
       ("symmetric", "constant") + ("zerograd",) * 4]


def _problem(n, k, rec, lim, rs, st, nt, ng=3):
    bcc = np.tile(np.array([1.1, 0.1, 2.2, 0.3, 0.0]), (6, 1))
    p = P.Problem("run1d", 1, n, ng=ng, num_tracers=nt, dx=1.0 / n, bc=BCS[k % len(BCS)], bc_const=bcc,
                  reconstruction=rec, slope_limiter=lim, riemann_solver=rs, time_stepper=st, max_cfl=0.4,
                  max_time=1e30, output_delta=1e30, gravity=(-0.3, 0.0, 0.0) if k % 3 == 2 else None)
    p.Q = P.random_state(1, n, ng=ng, num_tracers=nt, seed=n + k, vmax=0.4)
    return p


@pytest.mark.parametrize("n", [3, 30, 31, 95, 1024, 3840, 3841, 7680, 7681])
def test_one_launch_loop_against_port(gpu_lib, oracle_port, n):
    from mosscap_b200.hydro import HydroSim
    for k, (rec, lim, rs, st, nt) in enumerate([("muscl", "minmod", "hllc", "rk2", 0),
                                                ("weno5z", "minmod", "hllc", "ssprk3", 1),
                                                ("ppm", "vanleer", "hll", "ssprk4", 0),
                                                ("fog", "minmod", "rusanov", "rk2", 2)]):
        p = _problem(n, k, rec, lim, rs, st, nt)
        sim = HydroSim(p)
        ref = oracle_port.OracleSim(oracle_port.OracleConfig(**p.scheme_fields()), "port")
        if p.gravity is not None:
            ref.set_gravity(p.gravity)
        ref.set_Q(p.Q)
        sim.fill_bcs()
        ref.fill_bcs()
        before = sim.launch_count()
        dts, rdts = sim.advance(7), ref.run(7)
        # the clock's set-up, the CFL minimum, its reset and the first dt, then the steps
        assert (sim.launch_count() - before == 5) == (n <= 7680)
        assert np.array_equal(dts.view(np.uint64), rdts.view(np.uint64)), (rec, n)
        q, r = sim.get_Q(), ref.get_Q()
        assert np.array_equal(q.view(np.uint64), r.view(np.uint64)), (rec, n, np.abs(q - r).max())
        assert sim.status() == 0
        assert np.array_equal(sim.get_W().view(np.uint64), ref.get_W().view(np.uint64)), (rec, n)
        # the clock goes on: one more call, then a step through the hooks
        dts, rdts = sim.run(3), ref.run(3)
        assert np.array_equal(dts.view(np.uint64), rdts.view(np.uint64))
        assert np.array_equal(sim.get_Q().view(np.uint64), ref.get_Q().view(np.uint64))
        assert sim.last_cfl_min() > 0.0


def test_one_launch_loop_stops_at_outputs(gpu_lib, oracle_port):
    from mosscap_b200.hydro import HydroSim
    p = P.sod_1d(400).with_scheme(max_time=0.05, output_delta=0.013)
    sim = HydroSim(p)
    ref = oracle_port.OracleSim(oracle_port.OracleConfig(**p.scheme_fields()), "port")
    ref.set_Q(p.Q)
    sim.fill_bcs()
    ref.fill_bcs()
    dts, rdts = sim.run(), ref.run(10 ** 6)
    assert np.array_equal(dts.view(np.uint64), rdts.view(np.uint64))
    assert np.array_equal(sim.get_Q().view(np.uint64), ref.get_Q().view(np.uint64))
    assert sim.time >= 0.05 and len(sim.advance(5)) == 0


@pytest.mark.parametrize("n", [31, 1000, 5000])
def test_one_launch_loop_fp32_matches_launches(gpu_lib, n):
    from mosscap_b200 import capi
    from mosscap_b200.hydro import HydroSim
    for k, (rec, lim, rs, st, nt) in enumerate([("muscl", "minmod", "hllc", "rk2", 0),
                                                ("weno5z", "minmod", "hllc", "ssprk3", 0),
                                                ("ppm", "monotonizedcentral", "hll", "ssprk4", 1)]):
        p = _problem(n, k, rec, lim, rs, st, nt)
        a, b = HydroSim(p, precision="fp32"), HydroSim(p, precision="fp32")
        a.fill_bcs()
        b.fill_bcs()
        hook = capi.CFL_REDUCE_FN(lambda user, bits, stream: None)
        capi.check(gpu_lib.mc_set_cfl_reduce_hook(b.ctx, hook, None), "hook")
        da, db = a.run(6), b.run(6)
        assert np.array_equal(da.view(np.uint64), db.view(np.uint64)), (rec, n)
        assert np.array_equal(a.get_Q().view(np.uint64), b.get_Q().view(np.uint64)), (rec, n)
        assert np.array_equal(a.get_W().view(np.uint64), b.get_W().view(np.uint64)), (rec, n)
