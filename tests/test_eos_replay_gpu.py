"""The analytic LTE hydrogen update replays its bisection from a bracket of the root; the
same cells with the function evaluated at every step give the same bits on the same device.
Cells over wide ranges, cells around the rule that refuses the bracket (where the rounding
error of the function is near the margin), and states outside the physics."""
import ctypes

import numpy as np
import pytest
import torch

from mosscap_b200 import problems as P

pytestmark = pytest.mark.gpu

N = 1 << 18
SAHA, T_ION, U = 2.4146830395719654e21, 157763.42386247337, 2.0 ** -53


def _cells(kind, ion, avg_mass, gamma, rng):
    """(rho, internal energy) of N cells."""
    if kind == "rule":
        # rounding error u t1 (1 + k) r / 4 from a tenth of the rule's limit to ten times it
        temp = 10.0 ** rng.uniform(3.6, 6.5, N)
        t1 = 2.0 * temp + (157803.4 * (gamma - 1.0) if ion else 0.0)
        amp = t1 + (157803.4 * (gamma - 1.0) if ion else 0.0)
        r = 10.0 ** rng.uniform(-1.0, 1.0, N) * 0.0045 * 4.0 / (U * amp)
        rho = SAHA * temp ** 1.5 * np.exp(-T_ION / temp) / r * P.H_MASS * avg_mass
    else:
        (d0, d1), (t0, t1) = {"wide": ((-16, -2), (2.5, 5.5)), "usual": ((-9, -6), (3.7, 4.3)),
                              "hot": ((-13, -9), (4.5, 6.5)), "dense": ((-6, 2), (2.0, 5.0))}[kind]
        rho, temp = 10.0 ** rng.uniform(d0, d1, N), 10.0 ** rng.uniform(t0, t1, N)
    return rho, P.lte_internal_energy(rho, temp, gamma, avg_mass, ion)


def _update(lib, q, gamma, avg_mass, ion, plain):
    from mosscap_b200 import capi
    out = torch.full((2, q.shape[1]), -7.0, dtype=torch.float64, device="cuda")
    capi.check(lib.mc_debug_lte_update(ctypes.c_void_p(q.data_ptr()), q.shape[1], gamma, avg_mass, int(ion), int(plain),
                                       ctypes.c_void_p(out[0].data_ptr()), ctypes.c_void_p(out[1].data_ptr()), None),
               "mc_debug_lte_update")
    torch.cuda.synchronize()
    return out.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("kind", ["rule", "wide", "usual", "hot", "dense", "outside"])
@pytest.mark.parametrize("ion", [False, True])
@pytest.mark.parametrize("avg_mass,gamma", [(1.0, 5.0 / 3.0), (1.3, 1.1)])
def test_replayed_bisection_gives_the_plain_bits(gpu_lib, kind, ion, avg_mass, gamma):
    rng = np.random.default_rng(11)
    q = np.zeros((3, N))
    if kind == "outside":
        special = [0.0, -0.0, 1e-320, -1e-7, 1e-300, 1e300, np.inf, -np.inf, np.nan, 1e-7, 1e-40, 1e40, 1e3]
        q[0] = rng.choice(special, N)
        q[2] = rng.choice(special, N)
    else:
        q[0], q[2] = _cells(kind, ion, avg_mass, gamma, rng)
        v = rng.uniform(-5e3, 5e3, N)
        q[1] = q[0] * v
        q[2] += 0.5 * q[0] * v * v
    qt = torch.tensor(q, device="cuda")
    got = _update(gpu_lib, qt, gamma, avg_mass, ion, False)
    want = _update(gpu_lib, qt, gamma, avg_mass, ion, True)
    bad = np.flatnonzero((got != want).any(0))
    if kind == "outside":  # a NaN's bits are free
        bad = bad[~np.isnan(got.view(np.float64)[:, bad]).any(0) | ~np.isnan(want.view(np.float64)[:, bad]).any(0)]
    assert bad.size == 0, (bad.size, q[:, bad[:3]], got.view(np.float64)[:, bad[:3]], want.view(np.float64)[:, bad[:3]])
