"""The work that programs built on this framework have it do, as cases to time.

Every case is one pass through the public entry points on inputs made from a
seed: a few time steps of :class:`HydroSim` in its three loops (the
device-driven loop, the compute_dt / time_step hooks, the host-resident
state), of :class:`BatchSim`, or a forward and backward pass of
:class:`EulerSteps`. Simulations go on from pass to pass, as in a run.

``exact`` evolves the same inputs with a plain torch float64 solver of the
same schemes (this file's own, whole-array operations); gradients come from
torch's autograd through it.
"""
import math

import numpy as np
import torch

from mosscap_b200.adjoint import EulerSteps
from mosscap_b200.hydro import BatchSim, HydroSim
from mosscap_b200.problems import H_MASS, K_B, Problem, saha_y

NG = 3
FAR = 1e30  # no output clock: a pass is a fixed number of steps


def grid(name, setup, nx, ny=1, nz=1, recon="muscl", limiter="monotonizedcentral", riemann="hllc",
         stepper="ssprk3", precision="fp64", loop="device", steps=1, tracers=0, gravity=False):
    return dict(name=name, kind="grid", setup=setup, nx=nx, ny=ny, nz=nz, recon=recon, limiter=limiter,
                riemann=riemann, stepper=stepper, precision=precision, loop=loop, steps=steps, tracers=tracers,
                gravity=gravity)


def listed():
    return [
        # a shock tube: the smallest problem, all launches and latency
        grid("tube_1024", "tube", 1024, limiter="minmod", stepper="rk2", steps=32),
        # a shear layer of a parameter study or a first look: a grid of about one wave of tiles
        grid("shear_256", "shear", 256, 256, recon="weno5z", steps=8),
        # the production resolution of the same problem, in both precisions
        grid("shear_2048", "shear", 2048, 2048, recon="weno5z", steps=2),
        grid("shear_2048_fp32", "shear", 2048, 2048, recon="weno5z", precision="fp32", steps=2),
        # a program that keeps its state in host memory between steps; ragged rows
        grid("shear_host_1535x1023", "shear", 1535, 1023, recon="weno5z", loop="host"),
        # the main loop of the reference through its two hooks: a stratified box
        # with walls, an open top, a tracer, gravity, odd extents
        grid("box_777x1031", "box", 777, 1031, recon="ppm", riemann="hll", stepper="rk2", loop="hooks", steps=2,
             tracers=1, gravity=True),
        # a blast wave in 3D, and a smaller one of odd extents in the FP32 form
        grid("blast_256", "blast", 256, 256, 256, recon="ppm", riemann="hll"),
        grid("blast_fp32_151x187x129", "blast", 151, 187, 129, recon="ppm", riemann="hll", precision="fp32", steps=2),
        # partially ionised hydrogen: the equation of state evaluated at every
        # stage, its fields read at the end of the pass
        grid("hydrogen_512", "hydrogen", 512, 512, steps=8),
        # an ensemble of independent problems of uneven size, in both precisions
        dict(name="batch_384", kind="batch", n1d=192, n2d=192, max1d=4096, max2d=512, riemann="hllc",
             precision="fp64", steps=4),
        dict(name="batch_384_fp32", kind="batch", n1d=192, n2d=192, max1d=4096, max2d=512, riemann="hllc",
             precision="fp32", steps=4),
        # gradients of a run: the forward pass and the discrete adjoint
        dict(name="adjoint_512", kind="adjoint", nx=512, ny=512, steps=20, every=10),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["1d", "2d", "2d", "shear", "host", "3d", "hydrogen", "batch", "batch", "adjoint"])
    scheme = dict(recon=rng.choice(["muscl", "ppm", "weno5z"]), limiter=rng.choice(["minmod", "monotonizedcentral", "vanleer"]),
                  riemann=rng.choice(["hllc", "hll", "rusanov"]), stepper=rng.choice(["rk2", "ssprk3"]))
    precision = rng.choice(["fp64", "fp64", "fp32"])
    if kind == "1d":
        c = grid("", "tube", size(64, 65536), steps=size(2, 32), precision=precision, **scheme)
    elif kind == "2d":
        c = grid("", "box", size(48, 1536), size(48, 1536), loop="hooks", steps=size(1, 3), precision=precision,
                 tracers=rng.choice([0, 0, 1, 2]), gravity=rng.random() < 0.5, **scheme)
    elif kind == "shear":
        c = grid("", "shear", size(64, 2048), size(64, 2048), recon="weno5z", precision=precision, steps=2)
    elif kind == "host":
        c = grid("", "shear", size(128, 1536), size(128, 1536), loop="host", precision=precision, **scheme)
    elif kind == "3d":
        c = grid("", "blast", size(24, 224), size(24, 224), size(24, 224), recon="ppm", riemann="hll",
                 precision=precision)
    elif kind == "hydrogen":
        c = grid("", "hydrogen", size(64, 768), size(64, 768), steps=size(1, 4))
    elif kind == "batch":
        c = dict(kind="batch", n1d=size(8, 256), n2d=size(8, 192), max1d=size(256, 4096), max2d=size(96, 512),
                 riemann=rng.choice(["hllc", "rusanov"]), precision=precision, steps=size(1, 4))
    else:
        every = rng.choice([5, 10])
        c = dict(kind="adjoint", nx=size(64, 512), ny=size(64, 512), steps=every * rng.choice([1, 2]), every=every)
    c.pop("name", None)
    return c


# ---- inputs ---------------------------------------------------------------------

GAMMA = {"tube": 1.4, "shear": 5.0 / 3.0, "box": 1.4, "blast": 1.4, "hydrogen": 5.0 / 3.0}
GRAVITY = (0.0, -0.1, 0.0)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _axis(n):
    """Cell centres in units of the extent, ghosts included."""
    return (torch.arange(n + 2 * NG, dtype=torch.float64, device="cuda") - NG + 0.5) / n


def _waves(gen, axes, amplitude=1.0):
    """A smooth random field over the axes: a few periodic modes, at most `amplitude`."""
    f = 0.0
    for _ in range(3):
        r = torch.rand(2 * len(axes) + 1, generator=gen, device="cuda", dtype=torch.float64)
        term = 0.3 + 0.7 * r[-1]
        for a, x in enumerate(axes):
            k = 1.0 + torch.floor(3.0 * r[2 * a])
            term = term * torch.sin(2.0 * math.pi * (k * x + r[2 * a + 1]))
        f = f + term
    return f * (amplitude / 3.0)


def _conserved(w, nd, gamma):
    q = torch.empty_like(w)
    q[0] = w[0]
    for a in range(nd):
        q[1 + a] = w[0] * w[1 + a]
    q[1 + nd] = w[1 + nd] / (gamma - 1.0) + 0.5 * w[0] * (w[1:1 + nd] ** 2).sum(0)
    for t in range(2 + nd, w.shape[0]):
        q[t] = w[0] * w[t]
    return q


def _initial(c, seed):
    """(Problem, conserved state on the GPU) of a grid case."""
    gen = _generator(seed)
    nd = 1 if c["ny"] == 1 else 2 if c["nz"] == 1 else 3
    setup, gamma = c["setup"], GAMMA[c["setup"]]
    n = (c["nx"], c["ny"], c["nz"])
    dx, bc, cfl = 1.0 / n[0], ("zerograd",) * 6, 0.4
    x = _axis(n[0])[None, None, :]
    y = _axis(n[1])[None, :, None] if nd > 1 else None
    z = _axis(n[2])[:, None, None] if nd > 2 else None
    shape = (2 + nd + c["tracers"],) + tuple(m + 2 * NG if a < nd else 1 for a, m in reversed(list(enumerate(n))))
    w = torch.zeros(shape, dtype=torch.float64, device="cuda")
    r = torch.rand(8, generator=gen, device="cuda", dtype=torch.float64)
    noise = lambda: 2.0 * torch.rand(shape[1:], generator=gen, device="cuda", dtype=torch.float64) - 1.0  # noqa: E731
    if setup == "tube":
        cfl = 0.8
        left = x < 0.4 + 0.2 * r[0]
        w[0] = torch.where(left, 0.8 + 0.4 * r[1], 0.1 + 0.1 * r[2])
        w[1] = torch.where(left, 0.2 * r[3], -0.2 * r[4])
        w[2] = torch.where(left, 0.8 + 0.4 * r[5], 0.05 + 0.1 * r[6])
    elif setup == "shear":
        # Kelvin-Helmholtz: a dense band moving against its surroundings
        bc = ("periodic",) * 6
        band = (y - 0.5).abs() < 0.25
        w[0] = torch.where(band, 2.0, 1.0)
        w[1] = torch.where(band, 0.5, -0.5)
        w[2] = 0.01 * torch.sin(4.0 * math.pi * x) + 1e-3 * noise()
        w[3] = 2.5
    elif setup == "box":
        bc = ("wall", "symmetric", "wall", "symmetricoutflowdiode", "zerograd", "zerograd")
        w[0] = (1.0 - 0.2 * y) * (1.0 + _waves(gen, (x, y), 0.2))
        w[1] = _waves(gen, (x, y), 0.3)
        w[2] = _waves(gen, (x, y), 0.3)
        w[3] = 1.0 + _waves(gen, (x, y), 0.2)
        for t in range(c["tracers"]):
            w[4 + t] = 0.5 + 0.4 * torch.tanh(8.0 * _waves(gen, (x, y)))
    elif setup == "blast":
        # a Sedov-style blast: the energy of the cells within three cells of the
        # centre, in a cold medium with small density fluctuations
        dx, cfl = 2.0 / n[0], 0.8 / 3.0
        r2 = ((x - 0.5) * n[0]) ** 2 + ((y - 0.5) * n[1]) ** 2 + ((z - 0.5) * n[2]) ** 2
        hot = r2 < 9.0
        w[0] = 1.0 + 0.01 * noise()
        w[4] = torch.where(hot, (gamma - 1.0) * (0.5 + r[0]) / (hot.sum() * dx ** 3), 1e-5)
    if setup == "hydrogen":
        bc, dx = ("periodic",) * 6, 1.0e4
        rho = 10.0 ** (-7.5 + _waves(gen, (x, y), 1.5))
        temp = 10.0 ** (4.0 + _waves(gen, (x, y), 0.3))
        frac = torch.from_numpy(saha_y((rho / H_MASS).cpu().numpy(), temp.cpu().numpy())).cuda()
        w[0] = rho
        w[1] = _waves(gen, (x, y), 5.0e3)
        w[2] = _waves(gen, (x, y), 5.0e3)
        w[3] = rho * (K_B / H_MASS) * (1.0 + frac) * temp
    p = Problem(setup, nd, c["nx"], c["ny"], c["nz"], ng=NG, num_tracers=c["tracers"], dx=dx, bc=bc,
                reconstruction=c["recon"], slope_limiter=c["limiter"], riemann_solver=c["riemann"],
                time_stepper=c["stepper"], gamma=gamma, max_cfl=cfl, max_time=FAR, output_delta=FAR,
                gravity=GRAVITY if c["gravity"] else None, eos="analyticlteh" if setup == "hydrogen" else "ideal")
    return p, _conserved(w, nd, gamma)


def _batch_problems(c, seed):
    """Shock tubes and four-quadrant problems, sizes log-uniform, with the
    states' pressures and densities over two decades and subsonic velocities."""
    rng = np.random.default_rng(seed)
    out = []
    # the sizes belong to the case, not to the seed: every state costs the same
    sizes = np.random.default_rng(12)

    def state(nd):
        rho, p = np.exp(rng.uniform(np.log(0.1), np.log(10.0), size=2))
        return rho, rng.uniform(-0.6, 0.6, size=nd) * np.sqrt(1.4 * p / rho), p

    for k in range(c["n1d"] + c["n2d"]):
        nd = 1 if k < c["n1d"] else 2
        n = int(round(np.exp(sizes.uniform(np.log(64), np.log(c["max1d"] if nd == 1 else c["max2d"])))))
        x = (np.arange(n + 2 * NG) - NG + 0.5) / n
        right = x >= 0.5
        region = right[None, :].astype(int) if nd == 1 else right[None, :] + 2 * right[:, None]
        w = np.empty((2 + nd, 1) + region.shape)
        for g in range(2 ** nd):
            rho, v, p = state(nd)
            for i, s in enumerate((rho, *v, p)):
                w[i, 0][region == g] = s
        q = w.copy()
        q[1:1 + nd] *= w[0]
        q[1 + nd] = w[1 + nd] / 0.4 + 0.5 * w[0] * (w[1:1 + nd] ** 2).sum(0)
        out.append(Problem("tube" if nd == 1 else "quadrants", nd, n, n if nd > 1 else 1, ng=NG, dx=1.0 / n,
                           bc=("zerograd",) * 6, reconstruction="muscl", slope_limiter="minmod",
                           riemann_solver=c["riemann"], time_stepper="rk2", gamma=1.4, max_cfl=0.8 / nd,
                           max_time=FAR, output_delta=FAR, Q=q))
    return out


def _adjoint_inputs(c, seed):
    """A smooth shear flow with fluctuations in every field, gamma, and the
    derivative of the loss at the end of the run."""
    gen = _generator(seed)
    gamma = 5.0 / 3.0
    x, y = _axis(c["nx"])[None, NG:-NG], _axis(c["ny"])[NG:-NG, None]
    shape = (c["ny"], c["nx"])
    w = torch.empty((4,) + shape, dtype=torch.float64, device="cuda")
    layer = torch.tanh((0.25 - (y - 0.5).abs()) / 0.05)
    for v, (base, amp) in enumerate(((1.5 + 0.5 * layer, 0.1), (0.5 * layer, 0.05), (0.0, 0.05), (2.5, 0.1))):
        fluct = 2.0 * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) - 1.0
        w[v] = base + _waves(gen, (x, y), amp) + 1e-3 * fluct
    p = Problem("shear", 2, c["nx"], c["ny"], ng=NG, dx=1.0 / c["nx"], bc=("periodic",) * 6,
                reconstruction="weno5z", riemann_solver="hllc", time_stepper="ssprk3", gamma=gamma, max_cfl=0.4,
                max_time=FAR, output_delta=FAR)
    g_out = torch.zeros_like(w)
    g_out[0] = _waves(gen, (x, y))
    return p, _conserved(w, 2, gamma), torch.tensor(gamma, dtype=torch.float64), g_out


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "batch":
        sim = BatchSim(_batch_problems(c, seed), precision=c["precision"])
        sim.fill_bcs()
        sim.tune()
        return dict(c=c, sim=sim)
    if c["kind"] == "adjoint":
        p, q, gamma, g_out = _adjoint_inputs(c, seed)
        return dict(c=c, p=p, q=q.requires_grad_(), gamma=gamma.requires_grad_(), g_out=g_out)
    p, q = _initial(c, seed)
    sim = HydroSim(p, precision=c["precision"], Q=q.cpu().numpy())
    sim.fill_bcs()
    s = dict(c=c, sim=sim)
    if c["loop"] == "host":
        s["host"] = sim.Q.cpu().pin_memory()
    return s


def run(state):
    c = state["c"]
    if c["kind"] == "batch":
        state["sim"].advance(c["steps"])
        return {"pool": state["sim"].pool}
    if c["kind"] == "adjoint":
        q = EulerSteps.apply(state["q"], state["gamma"], state["p"], c["steps"], c["every"])
        gq, gg = torch.autograd.grad(q, (state["q"], state["gamma"]), state["g_out"])
        return {"q": q.detach(), "grad_q": gq, "grad_gamma": gg}
    sim = state["sim"]
    if c["loop"] == "host":
        dts = [sim.step_host(state["host"]) for _ in range(c["steps"])]
        return {"q": state["host"], "dt": dts}
    if c["loop"] == "hooks":
        dts = []
        for _ in range(c["steps"]):
            dts.append(sim.compute_dt())
            sim.time_step(dts[-1])
        return {"q": sim.Q, "dt": dts}
    dts = sim.advance(c["steps"])
    out = {"q": sim.Q, "dt": dts}
    if c["setup"] == "hydrogen":
        out["ionisation"], out["temperature"] = sim.eos_fields()
    return out


# ---- what a pass needs ------------------------------------------------------------

STAGES = {"rk2": 2, "ssprk3": 3, "ssprk4": 4}
# arithmetic per variable and axis of a reconstruction, a division or root counted as one
RECON_OPS = {"fog": 0, "muscl": 10, "ppm": 40, "weno5z": 76}


def _cell_ops(nd, nvar, recon, riemann):
    face = {"rusanov": 60, "hll": 70, "hllc": 80}[riemann]
    return nd * (nvar * RECON_OPS[recon] + face) + 8 * nvar + 3 * nd + 5


def work(case):
    c = case
    if c["kind"] == "batch":
        flops = bytes_ = 0.0
        for p in _batch_problems(c, 0):
            bytes_ += 2 * 8 * np.prod(p.shape)
            flops += p.interior_cells * 2 * c["steps"] * _cell_ops(p.num_dim, 2 + p.num_dim, "muscl", c["riemann"])
        return {"bytes": float(bytes_), "flops": float(flops)}
    nd = 1 if c["ny"] == 1 else 2 if c.get("nz", 1) == 1 else 3
    cells = c["nx"] * c["ny"] * c.get("nz", 1)
    if c["kind"] == "adjoint":
        # the state in and out, the derivative in and the gradient out; every
        # operation forward once and at least twice backward
        return {"bytes": 4 * 4 * 8.0 * cells,
                "flops": 3.0 * cells * 3 * c["steps"] * _cell_ops(2, 4, "weno5z", "hllc")}
    nvar = 2 + nd + c["tracers"]
    flops = cells * STAGES[c["stepper"]] * c["steps"] * _cell_ops(nd, nvar, c["recon"], c["riemann"])
    fields = 2 if c["setup"] == "hydrogen" else 0
    return {"bytes": 8.0 * cells * (2 * nvar + fields), "flops": float(flops)}


# ---- the same in plain torch, in 64 bits -------------------------------------------

TINY = 1e-20
WENO_EPS = 1e-36


def _fill(q, nd, bc):
    """Ghost cells of q [var, z, y, x] axis by axis, x first."""
    for a in range(nd):
        d = 3 - a
        n = q.shape[d] - 2 * NG
        inner = q.narrow(d, NG, n)
        ends = []
        for end in (0, 1):
            kind = bc[2 * a + end]
            if kind == "periodic":
                ends.append(inner.narrow(d, n - NG if end == 0 else 0, NG))
                continue
            if kind == "zerograd":
                edge = inner.narrow(d, 0 if end == 0 else n - 1, 1)
                ends.append(torch.cat([edge] * NG, d))
                continue
            g = inner.narrow(d, 0 if end == 0 else n - NG, NG).flip(d)
            if kind == "wall":
                g = torch.cat([g[:1 + a], -g[1 + a:2 + a], g[2 + a:]])
            elif kind == "symmetricoutflowdiode":
                m = g[1 + a:2 + a].clamp(max=0.0) if end == 0 else g[1 + a:2 + a].clamp(min=0.0)
                e = g[1 + nd:2 + nd] - (m - g[1 + a:2 + a]) ** 2 / g[:1]
                g = torch.cat([g[:1 + a], m, g[2 + a:1 + nd], e, g[2 + nd:]])
            ends.append(g)
        q = torch.cat([ends[0], inner, ends[1]], d)
    return q


def _prims(q, nd, gamma):
    v = [q[1 + a] / q[0] for a in range(nd)]
    p = (gamma - 1.0) * (q[1 + nd] - 0.5 * q[0] * sum(u * u for u in v))
    return [q[0], *v, p] + [q[t] / q[0] for t in range(2 + nd, q.shape[0])]


def _limited(um, up, limiter):
    if limiter == "vanleer":
        ok = um * up > 0
        return torch.where(ok, 2.0 * um * up / torch.where(ok, um + up, 1.0), 0.0)
    # the sign of zero counts as positive (or negative), as copysign has it
    s = torch.copysign(torch.ones_like(um), um) + torch.copysign(torch.ones_like(up), up)
    least = torch.minimum(um.abs(), up.abs())
    if limiter == "minmod":
        return 0.5 * s * least
    return s * torch.minimum(least, 0.25 * (um + up).abs())


def _faces(s, recon, limiter):
    """The values at the low and the high face of the cell in the middle of s[0..4]."""
    c = s[2]
    if recon == "fog":
        return c, c
    if recon == "muscl":
        d = 0.5 * _limited(c - s[1], s[3] - c, limiter)
        return c - d, c + d
    if recon == "ppm":
        dm, d0, dp = (_limited(s[k] - s[k - 1], s[k + 1] - s[k], limiter) for k in (1, 2, 3))
        l = 0.5 * (s[1] + c) - (d0 - dm) / 6.0
        r = 0.5 * (c + s[3]) - (dp - d0) / 6.0
        flat = (r - c) * (c - l) <= 0
        l, r = torch.where(flat, c, l), torch.where(flat, c, r)
        r = torch.where((r - c).abs() >= 2.0 * (l - c).abs(), 3.0 * c - 2.0 * l, r)
        l = torch.where((l - c).abs() >= 2.0 * (r - c).abs(), 3.0 * c - 2.0 * r, l)
        return l, r
    k = 13.0 / 12.0
    b0 = k * (s[0] - 2.0 * s[1] + c) ** 2 + 0.25 * (s[0] - 4.0 * s[1] + 3.0 * c) ** 2
    b1 = k * (s[1] - 2.0 * c + s[3]) ** 2 + 0.25 * (s[1] - s[3]) ** 2
    b2 = k * (c - 2.0 * s[3] + s[4]) ** 2 + 0.25 * (3.0 * c - 4.0 * s[3] + s[4]) ** 2
    tau = (b0 - b2).abs()
    i0, i1, i2 = (1.0 + (tau / (b + WENO_EPS)) ** 2 for b in (b0, b1, b2))

    def side(a, b, d, e, j0, j2):
        # candidate parabolas of cells (a, b, c), (b, c, d) and (c, d, e) at the face towards a
        w0, w1, w2 = 3.0 * j0, 6.0 * i1, j2
        return ((2.0 * c + 5.0 * b - a) * w0 + (2.0 * b - d + 5.0 * c) * w1 + (11.0 * c + 2.0 * e - 7.0 * d) * w2) \
            / (6.0 * (w0 + w1 + w2))

    return side(s[0], s[1], s[3], s[4], i0, i2), side(s[4], s[3], s[1], s[0], i2, i0)


def _flux(wl, wr, nd, a, gamma, riemann):
    """Interface flux along axis a of the hydro variables."""
    tracers = slice(2 + nd, None)
    tl, tr = wl[tracers], wr[tracers]
    vl, vr, pl, pr = wl[1 + a], wr[1 + a], wl[1 + nd], wr[1 + nd]
    cl, cr = (gamma * pl / wl[0]).sqrt(), (gamma * pr / wr[0]).sqrt()

    def cons(w):
        kin = 0.5 * w[0] * sum(w[1 + b] ** 2 for b in range(nd))
        return [w[0]] + [w[0] * w[1 + b] for b in range(nd)] + [w[1 + nd] / (gamma - 1.0) + kin]

    def phys(w, q, v, p):
        f = [x * v for x in q]
        f[1 + a] = f[1 + a] + p
        f[1 + nd] = f[1 + nd] + p * v
        return f

    ql, qr = cons(wl), cons(wr)
    if riemann in ("rusanov", "hll"):
        fl, fr = phys(wl, ql, vl, pl), phys(wr, qr, vr, pr)
        if riemann == "rusanov":
            s = 0.5 * (cl + vl.abs() + cr + vr.abs())
            f = [0.5 * (x + y - s * (v - u)) for x, y, u, v in zip(fl, fr, ql, qr)]
        else:
            sl = torch.minimum(vl - cl, vr - cr).clamp(max=-TINY)
            # the high estimate takes the low side's velocity on both sides
            sr = torch.maximum(vl + cl, vl + cr).clamp(min=-TINY)
            f = [(sr * x - sl * y + sr * sl * (v - u)) / (sr - sl) for x, y, u, v in zip(fl, fr, ql, qr)]
    else:
        mid = 0.5 * (pl + pr + (vl - vr) * 0.5 * (wl[0] + wr[0]) * 0.5 * (cl + cr))
        g = (gamma + 1.0) / (2.0 * gamma)
        one = torch.ones_like(mid)
        kl = torch.where(mid <= pl, one, (1.0 + g * (torch.where(mid <= pl, pl, mid) / pl - 1.0)).sqrt())
        kr = torch.where(mid <= pr, one, (1.0 + g * (torch.where(mid <= pr, pr, mid) / pr - 1.0)).sqrt())
        al, ar = vl - cl * kl, vr + cr * kr
        bm, bp = al.clamp(max=-TINY), ar.clamp(min=TINY)
        ul, ur = vl - al, vr - ar
        el, er = pl + ul * ql[1 + a], pr + ur * qr[1 + a]
        ml, mr = wl[0] * ul, -(wr[0] * ur)
        am = (el - er) / (ml + mr)
        cp = ((ml * er + mr * el) / (ml + mr)).clamp(min=0.0)

        def outer(w, q, v, p, b):
            f = [x * (v - b) for x in q]
            f[1 + a] = f[1 + a] + p
            f[1 + nd] = f[1 + nd] + p * v
            return f

        fl, fr = outer(wl, ql, vl, pl, bm), outer(wr, qr, vr, pr, bp)
        low = am >= 0
        den = torch.where(low, am - bm, bp - am)
        out, star = torch.where(low, am, -am) / den, torch.where(low, -bm, bp) / den
        f = [out * torch.where(low, x, y) for x, y in zip(fl, fr)]
        f[1 + a] = f[1 + a] + star * cp
        f[1 + nd] = f[1 + nd] + star * cp * am
    return f + [f[0] * torch.where(f[0] >= 0, x, y) for x, y in zip(tl, tr)]


def _divergence(q, p, gamma):
    """dx times minus the flux divergence over the interior, [var, z, y, x]."""
    nd = p.num_dim
    w = _prims(q, nd, gamma)
    n = (p.nx, p.ny, p.nz)
    total = None
    for a in range(nd):
        d = 2 - a
        lines = []
        for u in w:
            for b in range(nd):
                if b != a:
                    u = u.narrow(2 - b, NG, n[b])
            lines.append(u)
        lo, hi = [], []
        for u in lines:
            s = [u.narrow(d, NG - 1 + k - 2, n[a] + 2) for k in range(5)]
            l, r = _faces(s, p.reconstruction, p.slope_limiter)
            hi.append(r.narrow(d, 0, n[a] + 1))
            lo.append(l.narrow(d, 1, n[a] + 1))
        f = _flux(hi, lo, nd, a, gamma, p.riemann_solver)
        div = torch.stack([x.narrow(d, 0, n[a]) - x.narrow(d, 1, n[a]) for x in f])
        total = div if total is None else total + div
    return total


def _inner(q, p):
    for b, n in enumerate((p.nx, p.ny, p.nz)[:p.num_dim]):
        q = q.narrow(3 - b, NG, n)
    return q


def _dt(q, p, gamma):
    w = _prims(q, p.num_dim, gamma)
    c = (gamma * w[1 + p.num_dim] / w[0]).sqrt()
    v = sum(u * u for u in w[1:1 + p.num_dim]).sqrt()
    return p.max_cfl * (p.dx / (c + v)).min()


def _step(q, p, gamma, dt):
    """One SSPRK step of the padded state q."""
    def stage(q_in, a, b, c):
        # a q + b (q_in + c dt L(q_in))
        u = _divergence(q_in, p, gamma) * (dt / p.dx)
        x = _inner(q_in, p)
        if p.gravity is not None:
            nd = p.num_dim
            g = [x[0] * 0.0] + [x[0] * p.gravity[k] for k in range(nd)]
            g.append(sum(x[1 + k] * p.gravity[k] for k in range(nd)))
            g += [x[0] * 0.0] * p.num_tracers
            u = u + torch.stack(g) * dt
        new = b * x + b * c * u
        if a:
            new = new + a * _inner(q, p)
        pad = []
        for k in range(p.num_dim):
            pad += [NG, NG]
        return _fill(torch.nn.functional.pad(new, pad), p.num_dim, p.bc)

    if p.time_stepper == "rk2":
        return stage(stage(q, 0.0, 1.0, 1.0), 0.5, 0.5, 1.0)
    q1 = stage(q, 0.0, 1.0, 1.0)
    q2 = stage(q1, 0.75, 0.25, 1.0)
    return stage(q2, 1.0 / 3.0, 2.0 / 3.0, 1.0)


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "batch":
        parts = []
        with torch.no_grad():
            for p in _batch_problems(c, seed):
                q = _fill(torch.from_numpy(p.Q).cuda(), p.num_dim, p.bc)
                for _ in range(c["steps"]):
                    q = _step(q, p, p.gamma, _dt(q, p, p.gamma))
                q = q.reshape(-1)
                parts.append(torch.nn.functional.pad(q, (0, -q.numel() % 32)))
        return {"pool": torch.cat(parts)}
    if c["kind"] == "adjoint":
        from torch.utils.checkpoint import checkpoint
        p, q0, gamma, g_out = _adjoint_inputs(c, seed)
        q0 = q0.requires_grad_()
        gamma = gamma.cuda().requires_grad_()
        q = _fill(torch.nn.functional.pad(q0[:, None], (NG, NG, NG, NG)), 2, p.bc)
        for _ in range(c["steps"]):
            q = checkpoint(lambda u, g: _step(u, p, g, _dt(u, p, g)), q, gamma, use_reentrant=False)
        q = q[:, 0, NG:-NG, NG:-NG]
        gq, gg = torch.autograd.grad(q, (q0, gamma), g_out)
        return {"q": q.detach(), "grad_q": gq, "grad_gamma": gg.cpu()}
    with torch.no_grad():
        p, q = _initial(c, seed)
        q = _fill(q, p.num_dim, p.bc)
        dts = []
        for _ in range(c["steps"]):
            dt = _dt(q, p, p.gamma)
            q = _step(q, p, p.gamma, dt)
            dts.append(float(dt))
    out = {"q": q, "dt": dts if c["loop"] != "device" else np.array(dts)}
    if c["setup"] == "hydrogen":
        out["ionisation"] = out["temperature"] = None
    return out
