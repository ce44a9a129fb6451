"""Both sides of the sizes up to which a 1D FP64 problem with tracers takes whole steps in one
launch, against the C restatement bit for bit."""
import numpy as np
import pytest

from mosscap_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rec,nt,segments", [("weno5z", 2, 196), ("weno5z", 5, 154), ("ppm", 5, 200), ("ppm", 4, 256),
                                             ("muscl", 5, 256)])
@pytest.mark.parametrize("more", [0, 1])
def test_one_launch_limit_with_tracers(gpu_lib, oracle_port, rec, nt, segments, more):
    from mosscap_b200.hydro import HydroSim
    n = 30 * segments + more
    p = P.Problem("limit", 1, n, num_tracers=nt, dx=1.0 / n, bc=("zerograd",) * 6, reconstruction=rec,
                  riemann_solver="hllc", time_stepper="ssprk3", max_cfl=0.4, max_time=1e30, output_delta=1e30)
    p.Q = P.random_state(1, n, num_tracers=nt, seed=n, vmax=0.4)
    sim = HydroSim(p)
    ref = oracle_port.OracleSim(oracle_port.OracleConfig(**p.scheme_fields()), "port")
    ref.set_Q(p.Q)
    sim.fill_bcs()
    ref.fill_bcs()
    before = sim.launch_count()
    dts, rdts = sim.advance(3), ref.run(3)
    assert (sim.launch_count() - before == 5) == (more == 0)
    assert np.array_equal(dts.view(np.uint64), rdts.view(np.uint64))
    assert np.array_equal(sim.get_Q().view(np.uint64), ref.get_Q().view(np.uint64))
