"""The branch-free quotients and roots of the FP64 stage kernels, and the rule
that takes a tile to them.

Operations: IEEE results on random operands and on the operands whose exact
result lies closest to a rounding boundary, enumerated from their definition
(the only ones the error bounds in csrc/exact_fp64.cuh leave open).

Rule: states in range, out of range (scaled beyond it, in whole or in some
cells) and with zero, tiny and denormal velocities, against the C restatement
bit for bit."""
import ctypes

import numpy as np
import pytest
import torch

from mosscap_b200 import problems as P

pytestmark = pytest.mark.gpu


def _run(lib, op, a, b=None):
    from mosscap_b200 import capi
    at = torch.tensor(a, device="cuda")
    bt = torch.tensor(b, device="cuda") if b is not None else None
    out = torch.empty_like(at)
    capi.check(lib.mc_debug_exact_ops(op, ctypes.c_void_p(at.data_ptr()),
                                      ctypes.c_void_p(bt.data_ptr()) if bt is not None else None,
                                      ctypes.c_void_p(out.data_ptr()), at.numel(), None), "mc_debug_exact_ops")
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _same(got, want):
    got, want = got + 0.0, want + 0.0
    bad = np.flatnonzero(got.view(np.uint64) != want.view(np.uint64))
    assert bad.size == 0, (bad.size, bad[:4], got[bad[:4]], want[bad[:4]])


def _hard_quotients():
    """(a, b) in [1, 2) with a / b < 1 at the least distance from a rounding
    boundary, 2^54 A - M B = +-1 with odd M: for b just below 2 and for random b;
    and a / b = 1 - 1 / B next to 1 - 3 2^-54."""
    rng = np.random.default_rng(1)
    bs = [2 ** 53 - k for k in range(1, 1 << 15, 2)] + [int(x) | 1 for x in rng.integers(2 ** 52, 2 ** 53, 20000)]
    out = []
    for B in bs:
        inv = pow(B, -1, 1 << 54)
        for j in (1, -1):
            M = (-j * inv) % (1 << 54)
            A = (M * B + j) >> 54
            assert (A << 54) - M * B == j
            if M >= 1 << 53 and A >= 1 << 52:
                out.append((A, B))
    B = (1 << 54) // 3
    out += [(B - 1, B), (B, B + 1)]
    a = np.array([x for x, _ in out], dtype=np.float64) * 2.0 ** -52
    return a, np.array([y for _, y in out], dtype=np.float64) * 2.0 ** -52


def test_quotients_equal_ieee_division(gpu_lib):
    rng = np.random.default_rng(0)
    n = 1 << 21
    b = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-120, 121, n)
    a = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-250, 251, n) * rng.choice([-1.0, 1.0], n)
    a[: n // 16] = b[: n // 16] * rng.integers(1, 1 << 20, n // 16)  # near and at exact quotients
    a[-8:] = [0.0, -0.0] * 4  # (compared as values: the sign of a zero is free)
    b[:6] = [1.0, np.nextafter(2.0, 1.0), np.nextafter(1.0, 2.0), 3.0, 0.4, 2.0 / 3.0]
    _same(_run(gpu_lib, 0, a, b), a / b)
    _same(_run(gpu_lib, 0, np.ones_like(b), b), 1.0 / b)
    a, b = _hard_quotients()
    assert a.size > 10000
    _same(_run(gpu_lib, 0, a, b), a / b)
    _same(_run(gpu_lib, 0, -a * 2.0 ** 200, b * 2.0 ** -60), -a / b * 2.0 ** 260)
    _same(_run(gpu_lib, 0, np.ones_like(b), b), 1.0 / b)


def _square_roots_mod(c, bits):
    """Every r in [0, 2^bits) with r^2 = c (mod 2^bits), c = 1 (mod 8)."""
    r = 1
    for k in range(3, bits):
        if (r * r - c) % (1 << (k + 1)):
            r += 1 << (k - 1)
    assert (r * r - c) % (1 << bits) == 0
    half = 1 << (bits - 1)
    return {x % (1 << bits) for x in (r, -r, r + half, -r + half)}


def test_roots_equal_ieee_square_root(gpu_lib):
    rng = np.random.default_rng(2)
    n = 1 << 21
    x = rng.uniform(1.0, 4.0, n) * 4.0 ** rng.integers(-250, 251, n)
    x[: n // 16] = rng.integers(1, 1 << 26, n // 16).astype(np.float64) ** 2  # exact roots
    x[:4] = [1.0, np.nextafter(1.0, 2.0), np.nextafter(4.0, 1.0), 2.0]
    _same(_run(gpu_lib, 1, x), np.sqrt(x))
    # x = (M^2 + j) 2^-106 with odd M (a rounding boundary of the root) and odd j
    hard = []
    for bits, scale in ((54, 2.0 ** -52), (55, 2.0 ** -51)):  # x in [1, 2), x in [2, 4)
        for j in range(-255, 256, 2):
            if (-j) % 8 != 1:
                continue
            for r in _square_roots_mod(-j, bits):
                M = r
                while M < 1 << 54:
                    X = (M * M + j) >> bits
                    if M >= 1 << 53 and 1 << 52 <= X < 1 << 53:
                        hard.append(X * scale)
                    M += 1 << bits
    hard = np.array(hard)
    assert hard.size > 0
    for k in (0, 1, -100, 101):
        _same(_run(gpu_lib, 1, hard * 4.0 ** k), np.sqrt(hard * 4.0 ** k))


def _state(nd, n, kind, seed, nt):
    """A random state in, partly in or out of range."""
    nx, ny, nz = n
    q = P.random_state(nd, nx, ny, nz, num_tracers=nt, seed=seed, vmax=0.3)
    rng = np.random.default_rng(seed + 100)
    if kind == "scaled":
        q *= 1e-45  # rho, p below 2^-120 everywhere (velocities as they were)
    elif kind == "some":
        # a few cells whose density and pressure fall out of range
        for _ in range(3):
            at = tuple(int(rng.integers(0, m)) for m in q.shape[1:])
            q[(slice(None),) + at] *= 1e-37
    elif kind == "still":
        # zero, signed-zero, tiny and denormal velocities beside ordinary ones
        e_kin = 0.5 * (q[1:1 + nd] ** 2).sum(0) / q[0]
        e = q[1 + nd] - e_kin
        f = rng.choice([0.0, -0.0, 1e-90, 1e-310, 1.0], size=q[1:1 + nd].shape, p=[0.3, 0.2, 0.1, 0.1, 0.3])
        q[1:1 + nd] *= f
        q[1 + nd] = e + 0.5 * (q[1:1 + nd] ** 2).sum(0) / q[0]
    return q


@pytest.mark.parametrize("kind", ["in", "scaled", "some", "still"])
@pytest.mark.parametrize("nd,n,nt", [(1, (95, 1, 1), 1), (2, (61, 34, 1), 0), (2, (60, 46, 1), 2), (3, (36, 33, 31), 0)])
def test_range_rule_keeps_the_reference_bits(gpu_lib, oracle_port, kind, nd, n, nt):
    from mosscap_b200.hydro import HydroSim
    for k, (rec, lim, rs) in enumerate([("weno5z", "minmod", "hllc"), ("ppm", "monotonizedcentral", "hll"),
                                        ("muscl", "minmod", "hllc"), ("muscl", "vanleer", "rusanov"),
                                        ("ppm", "vanleer", "hllc"), ("muscl", "monotonizedcentral", "hll"),
                                        ("fog", "minmod", "hllc"), ("weno5z", "minmod", "rusanov")]):
        p = P.Problem("range", nd, *n, num_tracers=nt, dx=0.013, reconstruction=rec, slope_limiter=lim,
                      riemann_solver=rs, time_stepper="ssprk3" if k % 2 else "rk2", max_cfl=0.2, max_time=1e30,
                      output_delta=1e30, bc=("periodic", "periodic", "wall", "symmetric", "zerograd", "zerograd"))
        p.Q = _state(nd, n, kind, 7 * k + nd, nt)
        sim = HydroSim(p)
        ref = oracle_port.OracleSim(oracle_port.OracleConfig(**p.scheme_fields()), "port")
        ref.set_Q(p.Q)
        sim.fill_bcs()
        ref.fill_bcs()
        dts, rdts = sim.run(2), ref.run(2)
        what = (kind, rec, lim, rs)
        assert np.array_equal(dts.view(np.uint64), rdts.view(np.uint64)), what
        q, r = sim.get_Q(), ref.get_Q()
        assert np.isfinite(r).all(), what
        assert np.array_equal(q.view(np.uint64), r.view(np.uint64)), (what, np.abs(q - r).max())
