"""The work that a user of this framework has it do, as measurable cases.

Each case names one public entry point and its sizes:

  solve     CgSolver3D.solve: one pressure solve, system and right-hand side on the GPU
  precond   CgSolver3D.precond: one application of the MIC(0) preconditioner
  p2g, g2p  the particle/grid transfers
  substep   FluidSimulator: particles in, one substep, particles and pressure out
  frame     FluidSimulator: particles in, one CFL-limited frame, particles and pressure out
  grad      FlipLoss: forward and adjoint of a few differentiable substeps
  surface   sc_rebuild_surface_device: the fluid surface's triangle mesh, into the caller's buffers

listed() is the list, draw() gives further cases of the same ranges, prepare()
makes a case's inputs on the GPU, run() is one pass, work() the bytes and
operations the pass cannot do without, exact() the same outputs from plain torch
in 64 bits where there is such a value.
"""
import ctypes
import math

import torch

from simcraft_b200 import _capi, diff, fluid, solver

F64 = torch.float64


def listed():
    return [
        # The pressure solve of the smallest scene (32^3 cells), with the solver's own defaults
        # (absolute test, 1e-6): launches and latency.
        dict(name="solve_f64_32", kind="solve", nx=32, ny=32, nz=32, fill=0.5, precision="f64", criterion="abs", tol=1e-6,
             max_iter=300),
        # An odd, non-cubic domain to a tight tolerance.
        dict(name="solve_f64_ragged", kind="solve", nx=93, ny=50, nz=71, fill=0.5, precision="f64", criterion="rel",
             tol=1e-10, max_iter=2000),
        # The benchmark's standalone solve, in both precisions.
        dict(name="solve_f64_128", kind="solve", nx=128, ny=128, nz=128, fill=0.5, precision="f64", criterion="rel",
             tol=1e-8, max_iter=2000),
        dict(name="solve_mixed_128", kind="solve", nx=128, ny=128, nz=128, fill=0.5, precision="mixed", criterion="rel",
             tol=1e-8, max_iter=2000),
        # The same at the grid of the largest fluid scene.
        dict(name="solve_mixed_256", kind="solve", nx=256, ny=256, nz=256, fill=0.5, precision="mixed", criterion="rel",
             tol=1e-8, max_iter=2000),
        # The preconditioner alone, as an outer Krylov method of a caller's own applies it.
        dict(name="precond_f64", kind="precond", nx=160, ny=96, nz=128, fill=0.5),
        # The transfers as stages of a caller's own substep: particles of a dam break.
        dict(name="p2g_f64_128", kind="p2g", nx=128, ny=128, nz=128, fx=0.5, fy=0.5, ppc=8, flip=True),
        dict(name="g2p_f64_96", kind="g2p", nx=96, ny=96, nz=96, fx=0.5, fy=0.5, ppc=8, flip=True),
        # A small scene interactively: a frame of the 32^3 FP64 dam break.
        dict(name="frame_f64_32", kind="frame", n=32, fx=0.5, fy=0.5, ppc=8, precision="f64", advection="flip",
             criterion="rel", tol=1e-6, max_iter=200, tau=0.97, pcg="f64"),
        # The largest scene: a substep of the 256^3 FP32 dam break, 33.5M particles, mixed solve.
        dict(name="substep_f32_256", kind="substep", n=256, fx=0.5, fy=0.5, ppc=8, precision="f32", advection="flip",
             criterion="rel", tol=1e-8, max_iter=5000, tau=0.0, pcg="mixed"),
        # One gradient of the control problem: forward and adjoint.
        dict(name="grad_f64_48", kind="grad", n=48, steps=4, ppc=8, precision="f64", checkpoint_every=2),
        # The export of a frame's surface.
        dict(name="surface_192", kind="surface", nx=192, ny=192, nz=192),
    ]


def draw(rng):
    """One more case: a kind, then sizes spread over the logarithm of their range."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "precond", "p2g", "g2p", "frame", "substep", "grad", "surface"])
    if kind == "solve":
        m = size(24, 224)
        dims = [max(16, int(round(m * rng.uniform(0.6, 1.0)))) for _ in range(3)]
        dims[rng.randrange(3)] = m
        precision = rng.choice(["f64", "mixed"])
        if rng.random() < 0.25:
            crit, tol = "abs", 1e-6
        else:
            crit, tol = "rel", rng.choice([1e-6, 1e-8, 1e-10])
        return dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], fill=round(rng.uniform(0.35, 0.65), 3), precision=precision,
                    criterion=crit, tol=tol, max_iter=2000)
    if kind == "precond":
        return dict(kind=kind, nx=size(24, 192), ny=size(24, 192), nz=size(24, 192), fill=round(rng.uniform(0.35, 0.65), 3))
    if kind in ("p2g", "g2p"):
        return dict(kind=kind, nx=size(24, 144), ny=size(24, 144), nz=size(24, 144), fx=round(rng.uniform(0.3, 1.0), 3),
                    fy=round(rng.uniform(0.25, 0.6), 3), ppc=rng.choice([4, 8]), flip=rng.random() < 0.7)
    if kind in ("frame", "substep"):
        n = size(20, 40) if kind == "frame" else size(40, 160)
        precision = rng.choice(["f64", "f32"])
        tol = 1e-6 if kind == "frame" else 1e-8
        return dict(kind=kind, n=n, fx=round(rng.uniform(0.3, 1.0), 3), fy=round(rng.uniform(0.25, 0.6), 3),
                    ppc=rng.choice([4, 8]), precision=precision, advection=rng.choice(["flip", "flip", "pic"]), criterion="rel",
                    tol=tol, max_iter=5000, tau=0.0, pcg="mixed" if precision == "f32" else "f64")
    if kind == "grad":
        return dict(kind=kind, n=size(16, 56), steps=rng.choice([2, 3, 4]), ppc=8, precision="f64",
                    checkpoint_every=rng.choice([1, 2, 4]))
    return dict(kind=kind, nx=size(32, 224), ny=size(32, 224), nz=size(32, 224))


# ---------------------------------------------------------------------------
# Inputs

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=g.device, dtype=F64)


def _centres(n, h, dev):
    return (torch.arange(n, device=dev, dtype=F64) + 0.5) * h


def _sphere_sdf(dims, h, centres, radii, dev):
    x, y, z = (_centres(n, h, dev) for n in dims)
    best = torch.full(dims, math.inf, dtype=F64, device=dev)
    for c, r in zip(centres, radii):
        d2 = ((x - c[0]) ** 2)[:, None, None] + ((y - c[1]) ** 2)[None, :, None] + ((z - c[2]) ** 2)[None, None, :]
        torch.minimum(best, d2.sqrt_().sub_(r), out=best)
    return best


def _sphere_pool(dims, fill, seed, dev):
    """SDF of 24 spheres whose radii are scaled until they fill `fill` of the box, and the cell size."""
    g = _gen(seed, dev)
    m = max(dims)
    h = 1.0 / m
    ext = torch.tensor([n * h for n in dims], dtype=F64, device=dev)
    centres = (_rand(g, 24, 3) * ext).tolist()
    radii = (0.05 + 0.15 * _rand(g, 24)).tolist()
    probe = tuple(max(8, n * 48 // m) for n in dims)
    lo, hi = 0.2, 5.0
    for _ in range(12):
        mid = 0.5 * (lo + hi)
        f = float((_sphere_sdf(probe, 1.0 / max(probe), centres, [r * mid for r in radii], dev) <= 0).double().mean())
        lo, hi = (mid, hi) if f < fill else (lo, mid)
    return _sphere_sdf(dims, h, centres, [r * 0.5 * (lo + hi) for r in radii], dev), g


def _system(dims, fill, seed):
    """The pressure system of a sphere pool in a closed box, by the ghost-fluid rules: diagonal, the six
    couplings in the order Left, Right, Up, Down, Front, Back, right-hand side, active flags."""
    dev = _device()
    phi, g = _sphere_pool(dims, fill, seed, dev)
    factor = 32.0 / 120.0
    act = phi <= 0
    diag = torch.zeros(dims, dtype=F64, device=dev)
    pair = {}
    for axis in range(3):
        n = dims[axis]
        lo, hi = phi.narrow(axis, 0, n - 1), phi.narrow(axis, 1, n - 1)
        la, ha = lo <= 0, hi <= 0
        both = la & ha
        down, up = torch.zeros_like(diag), torch.zeros_like(diag)
        c = torch.where(both, -factor, 0.0)
        up.narrow(axis, 0, n - 1).copy_(c)
        down.narrow(axis, 1, n - 1).copy_(c)
        theta = (lo / (lo - hi)).clamp(0.01, 0.99)
        diag.narrow(axis, 0, n - 1).add_(torch.where(both, factor, torch.where(la & ~ha, factor / theta, 0.0)))
        diag.narrow(axis, 1, n - 1).add_(torch.where(both, factor, torch.where(ha & ~la, factor / (1.0 - theta), 0.0)))
        pair[axis] = (down, up)
    rhs = torch.where(act, _rand(g, *dims) * 2 - 1, 0.0)
    an = [pair[0][0], pair[0][1], pair[1][1], pair[1][0], pair[2][1], pair[2][0]]
    return diag, an, rhs, act.to(torch.uint8)


def _modes(g, k=4):
    return (_rand(g, k, 3, 3) * 2 - 1) * 6.0, _rand(g, k, 3) * 2 * math.pi


def _field(modes, x, a):
    """Component a of a smooth velocity field of magnitude below 1 at the points x (..., 3)."""
    k, ph = modes
    return sum(torch.sin(x @ k[i, a] + ph[i, a]) for i in range(k.shape[0])) / k.shape[0]


def _particles(dims, h, fx, fy, ppc, seed):
    """`ppc` particles jittered in every cell of a dam-break block, with a smooth velocity."""
    dev = _device()
    g = _gen(seed, dev)
    cx, cy, cz = max(1, round(fx * dims[0])), max(1, round(fy * dims[1])), dims[2]
    grid = torch.stack(torch.meshgrid(*(torch.arange(c, device=dev, dtype=F64) for c in (cx, cy, cz)), indexing="ij"), -1)
    pos = (grid.reshape(-1, 1, 3) + _rand(g, cx * cy * cz, ppc, 3)).reshape(-1, 3) * h
    del grid
    m = _modes(g)
    vel = torch.stack([_field(m, pos, a) for a in range(3)], -1)
    return pos.contiguous(), vel.contiguous(), g


def _faces(dims, h, g):
    """A smooth face velocity field and a perturbed one, as before and after a projection."""
    m, d = _modes(g), _modes(g)
    out = []
    for a, shape in enumerate(fluid.face_shapes(*dims)):
        ax = [(torch.arange(n, device=g.device, dtype=F64) + (0.0 if i == a else 0.5)) * h for i, n in enumerate(shape)]
        x = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1)
        now = _field(m, x, a).contiguous()
        out.append((now, (now + 0.1 * _field(d, x, a)).contiguous()))
    return [o[0] for o in out], [o[1] for o in out]


def _sim(case, n):
    res = (case["n"],) * 3
    return fluid.FluidSimulator(n, (1.0, 1.0, 1.0), res, precision=case["precision"], advection=case["advection"],
                                flip_alpha=0.95, cfl_factor=1.0, pcg_tol=case["tol"], pcg_max_iter=case["max_iter"],
                                pcg_criterion=solver.CRIT_REL_L2, pcg_mic_tau=case["tau"],
                                pcg_precision=solver.PREC_MIXED if case["pcg"] == "mixed" else solver.PREC_FP64)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "precond"):
        dims = (case["nx"], case["ny"], case["nz"])
        diag, an, rhs, act = _system(dims, case["fill"], seed)
        if kind == "precond":
            s = solver.CgSolver3D(*dims)
            torch.cuda.synchronize()
            s.upload(diag, an, rhs, act)
            return dict(kind=kind, s=s, r=rhs, z=torch.zeros_like(rhs))
        s = solver.CgSolver3D(*dims, tol=case["tol"], max_iter=case["max_iter"],
                              criterion=solver.CRIT_ABS_LINF if case["criterion"] == "abs" else solver.CRIT_REL_L2,
                              precision=solver.PREC_MIXED if case["precision"] == "mixed" else solver.PREC_FP64)
        return dict(kind=kind, s=s, diag=diag, an=an, rhs=rhs, act=act, p=torch.zeros_like(rhs))
    if kind in ("p2g", "g2p"):
        dims = (case["nx"], case["ny"], case["nz"])
        h = 1.0 / max(dims)
        pos, vel, g = _particles(dims, h, case["fx"], case["fy"], case["ppc"], seed)
        st = dict(kind=kind, dims=dims, h=h, pos=pos, vel=vel, flip=case["flip"])
        if kind == "g2p":
            st["last"], st["now"] = _faces(dims, h, g)
        return st
    if kind in ("frame", "substep"):
        n = case["n"]
        pos, vel, _ = _particles((n, n, n), 1.0 / n, case["fx"], case["fy"], case["ppc"], seed)
        sim = _sim(case, pos.shape[0])
        out = [torch.empty_like(pos), torch.empty_like(vel), torch.empty((n, n, n), dtype=F64, device=pos.device)]
        return dict(kind=kind, sim=sim, pos=pos, vel=vel, dt=1.0 / n if kind == "substep" else 1.0 / 120.0, out=out,
                    dtype=torch.float32 if case["precision"] == "f32" else F64)
    if kind == "grad":
        n = case["n"]
        pos, param, target, h = diff.control_scene(n, seed_particles=seed, seed_param=seed + 1, seed_target=seed + 2,
                                                   ppc=case["ppc"])
        sim = diff.DiffFlip((n, n, n), h, 1.0 / 120.0, case["steps"], precision=case["precision"],
                            checkpoint_every=case["checkpoint_every"], flip_alpha=0.95)
        sim.set_particles(pos)
        sim.set_target(target)
        return dict(kind=kind, sim=sim, param=torch.from_numpy(param).to(_device()).requires_grad_())
    dims = (case["nx"], case["ny"], case["nz"])
    phi, g = _sphere_pool(dims, 0.4, seed, _device())
    # a simulated surface is not smooth below the cell size
    phi += (0.1 / max(dims)) * (_rand(g, *dims) - 0.5)
    cap = 8 * (dims[0] * dims[1] + dims[1] * dims[2] + dims[0] * dims[2])
    mesh = dict(vertices=torch.zeros(cap, 3, dtype=F64, device=phi.device), normals=torch.zeros(cap, 3, dtype=F64, device=phi.device),
                indices=torch.zeros(6 * cap, dtype=torch.int32, device=phi.device))
    return dict(kind=kind, phi=phi, h=1.0 / max(dims), mesh=mesh, ctx=solver.default_context())


# ---------------------------------------------------------------------------
# One pass

def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(st):
    kind = st["kind"]
    if kind == "solve":
        st["s"].solve(st["diag"], st["an"], st["rhs"], st["act"], st["p"])
        return {"pressure": st["p"]}
    if kind == "precond":
        return {"z": st["s"].precond(st["r"], st["z"])}
    if kind == "p2g":
        return fluid.p2g(st["pos"], st["vel"], st["dims"], st["h"], flip=st["flip"])
    if kind == "g2p":
        if st["flip"]:
            return {"vel": fluid.g2p(st["pos"], st["vel"], st["dims"], st["h"], *st["now"], *st["last"], alpha=0.95)}
        return {"vel": fluid.g2p(st["pos"], st["vel"], st["dims"], st["h"], *st["now"], alpha=-1.0)}
    if kind in ("frame", "substep"):
        sim, (pos, vel, p) = st["sim"], st["out"]
        sim.set_initial_fluid(st["pos"], st["vel"])
        if kind == "substep":
            sim.substep(st["dt"])
        else:
            sim.step(st["dt"])
        # read back into device arrays through the C interface, as an engine that keeps its data on the GPU does
        L, check = _capi.lib(), _capi.check
        check("sc_fluid_get_particles", L.sc_fluid_get_particles(sim.handle, _ptr(pos), _ptr(vel), 1), sim.ctx.handle)
        check("sc_fluid_get_pressure", L.sc_fluid_get_pressure(sim.handle, _ptr(p), 1), sim.ctx.handle)
        sim.ctx.synchronize()
        return {"pos": pos.to(st["dtype"]), "vel": vel.to(st["dtype"]), "pressure": p.to(st["dtype"])}
    if kind == "grad":
        st["param"].grad = None
        loss = diff.FlipLoss.apply(st["param"], st["sim"])
        loss.backward()
        return {"loss": loss.detach(), "grad": st["param"].grad}
    # into buffers of a fixed size, as a renderer that keeps its vertex and index buffers does
    ctx, phi, mesh = st["ctx"], st["phi"], st["mesh"]
    spacing, origin = (ctypes.c_double * 3)(*[st["h"]] * 3), (ctypes.c_double * 3)()
    nv, ni = ctypes.c_int64(0), ctypes.c_int64(0)
    ctx.set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    try:
        _capi.check("sc_rebuild_surface_device", _capi.lib().sc_rebuild_surface_device(
            ctx.handle, *phi.shape, spacing, origin, _ptr(phi), _ptr(mesh["vertices"]), _ptr(mesh["normals"]),
            _ptr(mesh["indices"]), mesh["vertices"].shape[0], mesh["indices"].shape[0], ctypes.byref(nv), ctypes.byref(ni)),
            ctx.handle)
    finally:
        ctx.use_own_stream()
    return dict(mesh, counts=torch.tensor([nv.value, ni.value]))


# ---------------------------------------------------------------------------
# What a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind in ("solve", "precond"):
        n = case["nx"] * case["ny"] * case["nz"]
        if kind == "precond":
            # one read of the residual and of the factor (pivot and three couplings), one write
            return {"bytes": n * 8.0 * 6, "flops": n * case["fill"] * 16.0}
        # iterations grow with the longest side and the digits asked for; an iteration reads the matrix, the factor
        # and its vectors once
        digits = -math.log10(case["tol"])
        it = 0.11 * max(case["nx"], case["ny"], case["nz"]) * digits
        per = 4.0 * 17 if case["precision"] == "mixed" else 8.0 * 14
        return {"bytes": n * (8.0 * 7 + it * per), "flops": n * case["fill"] * it * 45.0}
    if kind in ("p2g", "g2p"):
        n = case["nx"] * case["ny"] * case["nz"]
        p = round(case["fx"] * case["nx"]) * round(case["fy"] * case["ny"]) * case["nz"] * case["ppc"]
        if kind == "p2g":
            return {"bytes": p * 48.0 + n * 3 * (25.0 if case["flip"] else 17.0), "flops": p * 3 * 64 * 4.0}
        return {"bytes": p * 72.0 + n * 3 * (16.0 if case["flip"] else 8.0), "flops": p * (6 if case["flip"] else 3) * 64 * 4.0}
    if kind in ("frame", "substep"):
        n = float(case["n"]) ** 3
        p = round(case["fx"] * case["n"]) * round(case["fy"] * case["n"]) * case["n"] * case["ppc"]
        it = 0.11 * case["n"] * -math.log10(case["tol"])
        fluid_part = case["fx"] * case["fy"]
        per = 4.0 * 17 if case["pcg"] == "mixed" else 8.0 * 14
        return {"bytes": p * 12 * 8.0 + n * 20 * 8.0 + n * fluid_part * it * per,
                "flops": n * fluid_part * it * 45.0 + p * 9 * 64 * 4.0}
    if kind == "grad":
        n, p = float(case["n"]) ** 3, 0.25 * case["n"] ** 3 * case["ppc"]
        it = 0.11 * case["n"] * 10
        # each substep is run forward and its adjoint back, each with one solve of the fluid quarter
        return {"bytes": 2 * case["steps"] * (n * 0.25 * it * 8.0 * 14 + p * 96.0 + n * 160.0),
                "flops": 2 * case["steps"] * n * 0.25 * it * 45.0}
    n = case["nx"] * case["ny"] * case["nz"]
    area = (case["nx"] * case["ny"] * case["nz"]) ** (2.0 / 3.0)
    return {"bytes": n * 8.0 + area * 5 * 60.0, "flops": n * 2.0}


# ---------------------------------------------------------------------------
# The same outputs from plain torch in 64 bits

def _apply(diag, an, x):
    y = diag * x
    for axis, lo, hi in ((0, an[0], an[1]), (1, an[3], an[2]), (2, an[5], an[4])):
        n = x.shape[axis]
        if n < 2:
            continue
        y.narrow(axis, 1, n - 1).addcmul_(lo.narrow(axis, 1, n - 1), x.narrow(axis, 0, n - 1))
        y.narrow(axis, 0, n - 1).addcmul_(hi.narrow(axis, 0, n - 1), x.narrow(axis, 1, n - 1))
    return y


def _exact_solve(case, seed):
    diag, an, rhs, act = _system((case["nx"], case["ny"], case["nz"]), case["fill"], seed)
    on = act.bool()
    inv = torch.where(on, 1.0 / torch.where(on, diag, 1.0), 0.0)
    x, goal = torch.zeros_like(rhs), 1e-13 * float(rhs.norm())
    r = rhs.clone()
    for _ in range(4):  # conjugate gradients, restarted on the true residual
        z = inv * r
        s, rho = z.clone(), (r * z).sum()
        for it in range(20 * max(rhs.shape)):
            q = _apply(diag, an, s)
            a = rho / (s * q).sum()
            x.addcmul_(a, s)
            r.addcmul_(-a, q)
            if it % 16 == 0 and float(r.norm()) < goal:
                break
            z = inv * r
            new = (r * z).sum()
            s = z + (new / rho) * s
            rho = new
        r = rhs - _apply(diag, an, x)
        if float(r.norm()) < 4 * goal:
            break
    return {"pressure": x}


def _exact_precond(case, seed, tau=0.97, sigma=0.25):
    """MIC(0) with the framework's pivot rule, plane by plane of constant i + j + k."""
    dims = (case["nx"], case["ny"], case["nz"])
    diag, an, rhs, act = _system(dims, case["fill"], seed)
    dev = diag.device
    pad = lambda t: torch.nn.functional.pad(t, (1, 1, 1, 1, 1, 1))  # noqa: E731
    A = torch.where(act.bool(), diag, 0.0)
    L, D, B = (pad(an[i]).reshape(-1) for i in (0, 3, 5))
    on = pad(act.double()).reshape(-1)
    A, r = pad(A).reshape(-1), pad(torch.where(act.bool(), rhs, 0.0)).reshape(-1)
    sy, sx = dims[2] + 2, (dims[1] + 2) * (dims[2] + 2)
    i, j, k = torch.meshgrid(*(torch.arange(1, n + 1, device=dev) for n in dims), indexing="ij")
    at = (i * sx + j * sy + k).reshape(-1)
    level, order = (i + j + k).reshape(-1).sort()
    order, cuts = at[order], torch.bincount(level).cumsum(0).tolist()
    planes = [order[a:b] for a, b in zip([0] + cuts[:-1], cuts) if b > a]
    step = {"x": sx, "y": sy, "z": 1}
    E = torch.zeros_like(A)
    terms = ((L, "x", "y", "z"), (D, "y", "x", "z"), (B, "z", "x", "y"))
    for p in planes:
        e = A[p].clone()
        for M, a, b, c in terms:
            q = p - step[a]
            Eq, m = E[q], M[p]
            ok = Eq != 0
            side = tau * m * (on[q + step[b]] * M[q + step[b]] + on[q + step[c]] * M[q + step[c]])
            e = e - torch.where(ok, (m * Eq) ** 2 + side / torch.where(ok, Eq * Eq, 1.0), 0.0)
        e = torch.where(e < sigma * A[p], A[p], e)
        E[p] = torch.where(A[p] != 0, 1.0 / torch.where(A[p] != 0, e, 1.0).sqrt(), 0.0)
    q = torch.zeros_like(A)
    for p in planes:
        t = r[p]
        for M, a, _, _ in terms:
            n = p - step[a]
            t = t - M[p] * E[n] * q[n]
        q[p] = t * E[p]
    z = torch.zeros_like(A)
    for p in reversed(planes):
        t = q[p]
        for M, a, _, _ in terms:
            n = p + step[a]
            t = t - M[n] * E[p] * z[n]
        z[p] = t * E[p]
    return {"z": z.reshape(tuple(n + 2 for n in dims))[1:-1, 1:-1, 1:-1].contiguous()}


def _spline(r):
    return torch.where(r < 1, 2.0 / 3.0 - r * r + 0.5 * r * r * r, (2.0 - r).clamp(min=0.0) ** 3 / 6.0)


def _nodes(pos, a, h):
    """Per axis: first node of the 4-node stencil and its factors, for face grid a."""
    base, w = [], []
    h = torch.tensor(h, dtype=F64, device=pos.device)  # on the GPU: division by a host number multiplies by its inverse
    for i in range(3):
        off = 0.0 if i == a else 0.5
        p = pos[:, i]
        b = ((p - off * h) / h + 0.5).to(torch.int64) - 1
        base.append(b)
        w.append([_spline((p - ((b + d).to(F64) + off) * h).abs() / h) for d in range(4)])
    return base, w


def _stencil(pos, a, dims, h):
    """Flat node index (0 where outside) and weight (0 where outside) of each of the 64 nodes in turn."""
    shape = fluid.face_shapes(*dims)[a]
    base, w = _nodes(pos, a, h)
    for i in range(4):
        for j in range(4):
            wij = w[0][i] * w[1][j]
            for k in range(4):
                n = [base[0] + i, base[1] + j, base[2] + k]
                ok = (n[0] >= 0) & (n[0] < shape[0]) & (n[1] >= 0) & (n[1] < shape[1]) & (n[2] >= 0) & (n[2] < shape[2])
                flat = (n[0] * shape[1] + n[1]) * shape[2] + n[2]
                yield torch.where(ok, flat, 0), torch.where(ok, wij * w[2][k], 0.0)


def _exact_p2g(case, seed):
    st = prepare(case, seed)
    out = {}
    for a, (name, shape) in enumerate(zip("uvw", fluid.face_shapes(*st["dims"]))):
        V = torch.zeros(math.prod(shape), dtype=F64, device=st["pos"].device)
        W = torch.zeros_like(V)
        for at, w in _stencil(st["pos"], a, st["dims"], st["h"]):
            V.index_add_(0, at, w * st["vel"][:, a])
            W.index_add_(0, at, w)
        ok = W > 0
        out[name] = torch.where(ok, V / torch.where(ok, W, 1.0), 0.0).reshape(shape)
        out[name + "w"] = W.reshape(shape)
        out[name + "valid"] = None
        if st["flip"]:
            out[name + "last"] = out[name]
    return out


def _exact_g2p(case, seed):
    st = prepare(case, seed)
    cols = []
    for a in range(3):
        def sample(g):
            s, ws = torch.zeros_like(st["pos"][:, 0]), torch.zeros_like(st["pos"][:, 0])
            for at, w in _stencil(st["pos"], a, st["dims"], st["h"]):
                s += g.reshape(-1)[at] * w
                ws += w
            return torch.where(ws > 0, s / torch.where(ws > 0, ws, 1.0), 0.0)

        now = sample(st["now"][a])
        cols.append(now + 0.95 * (st["vel"][:, a] - sample(st["last"][a])) if st["flip"] else now)
    return {"vel": torch.stack(cols, -1)}


def exact(case, seed):
    """None for the simulator's steps and the gradient (whole chains of the stages above around an iterative
    solve), and for the mesh, whose vertex list is an order rather than a value."""
    kind = case["kind"]
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind == "precond":
        return _exact_precond(case, seed)
    if kind == "p2g":
        return _exact_p2g(case, seed)
    if kind == "g2p":
        return _exact_g2p(case, seed)
    return None
