"""The 2D tile kernels on both sides of the rule that gives small grids lower tiles
(at most 148 tiles, one per SM), with the MUSCL tile load in 2D and 3D and the loads of
several cells at a time, against the C
restatement bit for bit."""
import numpy as np
import pytest

from mosscap_b200 import problems as P

pytestmark = pytest.mark.gpu


# tiles of 30 x 30: 148 (full height), 185, one, three of 8 rows with a ragged end,
# 168 (just above the rule), 144 of 16 rows; odd row lengths take no tensor copy
@pytest.mark.parametrize("nx,ny", [(120, 1110), (121, 1110), (30, 29), (31, 17), (420, 359), (256, 250)])
@pytest.mark.parametrize("rec,rs,st,ng", [("weno5z", "hllc", "ssprk3", 3), ("muscl", "hllc", "rk2", 3),
                                          ("muscl", "hll", "ssprk3", 2), ("ppm", "hll", "ssprk4", 4),
                                          ("fog", "rusanov", "rk2", 1)])
def test_tile_heights_and_loads_against_port(gpu_lib, oracle_port, nx, ny, rec, rs, st, ng):
    from mosscap_b200.hydro import HydroSim
    p = P.Problem("tiles", 2, nx, ny, ng=ng, dx=0.01, reconstruction=rec, riemann_solver=rs, time_stepper=st,
                  max_cfl=0.2, max_time=1e30, output_delta=1e30, gravity=(0.1, -0.2, 0.0) if rs == "hll" else None,
                  bc=("wall", "symmetric", "zerograd", "symmetricoutflowdiode", "zerograd", "zerograd"))
    p.Q = P.random_state(2, nx, ny, ng=ng, seed=nx + ny, vmax=0.3)
    sim = HydroSim(p)
    ref = oracle_port.OracleSim(oracle_port.OracleConfig(**p.scheme_fields()), "port")
    if p.gravity is not None:
        ref.set_gravity(p.gravity)
    ref.set_Q(p.Q)
    sim.fill_bcs()
    ref.fill_bcs()
    dts, rdts = sim.run(2), ref.run(2)
    assert np.array_equal(dts.view(np.uint64), rdts.view(np.uint64))
    q, r = sim.get_Q(), ref.get_Q()
    assert np.array_equal(q.view(np.uint64), r.view(np.uint64)), np.abs(q - r).max()
    assert sim.status() == 0


@pytest.mark.parametrize("nx,ny,nz", [(46, 40, 13), (47, 33, 31)])
@pytest.mark.parametrize("lim,nt", [("minmod", 0), ("vanleer", 2)])
def test_muscl_plane_pass_against_port(gpu_lib, oracle_port, nx, ny, nz, lim, nt):
    from mosscap_b200.hydro import HydroSim
    p = P.Problem("tiles3", 3, nx, ny, nz, num_tracers=nt, dx=0.01, reconstruction="muscl", slope_limiter=lim,
                  riemann_solver="hllc", time_stepper="rk2", max_cfl=0.2, max_time=1e30, output_delta=1e30,
                  bc=("wall", "symmetric", "zerograd", "zerograd", "periodic", "periodic"))
    p.Q = P.random_state(3, nx, ny, nz, num_tracers=nt, seed=nx, vmax=0.3)
    sim = HydroSim(p)
    ref = oracle_port.OracleSim(oracle_port.OracleConfig(**p.scheme_fields()), "port")
    ref.set_Q(p.Q)
    sim.fill_bcs()
    ref.fill_bcs()
    dts, rdts = sim.run(2), ref.run(2)
    assert np.array_equal(dts.view(np.uint64), rdts.view(np.uint64))
    assert np.array_equal(sim.get_Q().view(np.uint64), ref.get_Q().view(np.uint64))
