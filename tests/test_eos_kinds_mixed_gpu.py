"""The analytic LTE hydrogen update where cells whose bisection is replayed from a bracket
share warps with cells that evaluate every step (fully ionised, cold and neutral, or
invalid): the others' temperatures as without them."""
import numpy as np
import pytest

from mosscap_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ion", [False, True])
def test_mixed_cells(gpu_lib, oracle_port, ion):
    from mosscap_b200.hydro import HydroSim
    p = P.lte_hydrogen(2, 96, seed=4, ionisation=ion)
    rng = np.random.default_rng(8)
    kind = rng.choice(5, size=p.Q.shape[1:], p=[0.6, 0.1, 0.1, 0.1, 0.1])
    for k, (rho, temp) in {1: (1e-12, 1e6), 2: (1e-6, 300.0), 3: (1e-15, 3e4), 4: (1e-7, -5e3)}.items():
        e = P.lte_internal_energy(np.array(rho), np.array(abs(temp)), p.gamma, 1.0, ion) * np.sign(temp)
        for v, x in enumerate((rho, 0.0, 0.0, float(e))):
            p.Q[v][kind == k] = x
    sim = HydroSim(p)
    sim.update_eos()
    y, T = sim.eos_fields()
    ref = oracle_port.OracleSim(oracle_port.OracleConfig(**p.scheme_fields()), "port")
    ref.set_eos(p.eos, p.eos_avg_mass, p.eos_ionisation, p.eos_table)
    q = p.Q.copy()
    for v, x in enumerate((1e-7, 0.0, 0.0, 1e3)):
        q[v][kind == 4] = x  # the reference aborts on a negative energy
    ref.set_Q(q)
    ref.update_eos()
    y_ref, T_ref = ref.eos_fields()
    ordinary = np.isin(kind.reshape(T.shape), (0, 2))
    dT = np.abs(T - T_ref)[ordinary]
    assert dT.max() <= 0.25  # a bisection may end on the other side of one halving
    assert (dT == 0.0).mean() > 0.95
    assert sim.status() & 0x10
