"""The work this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values. Its ``kind`` says which entry points it goes through:

``step``      one time step from a given state: device arrays in and out
              (``set_state_device``, ``step_async``, ``get_state_device``), or host arrays
              (``host``: ``pbf_set_state``, ``pbf_step``, ``pbf_get_state``), for one scene or a
              batch of uneven scenes (``scenes``), with a box or a triangle mesh as collider
``rollout``   ``autograd.rollout`` over a few steps and the gradient of a loss of its result
``adjoint``   ``adjoint_step_device``: a recorded step and its reverse
``surface``   the marching-cubes surface of the fluid, into host arrays
``render``    one path-traced frame of the fluid in a Cornell box, into host arrays

Particles start as lattice blocks of spacing ``s = h / ratio`` whose positions are moved by up
to ``jitter`` spacings: 0.008 is the configured scenes' initial state, 0.2 a fluid in motion.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from fluid_gb300 import pbf, render, scenes
from fluid_gb300.autograd import rollout
from fluid_gb300.params import PBF_FLAG_GRAPH, PBF_FLAG_STATS, PbfParams

_STEP = dict(kind="step", nx=16, ny=16, nz=16, h=0.1, ratio=2.0, jitter=0.008, speed=0.0, iters=4, scorr_n=4,
             blocks=1, scenes=0, lo=0, hi=0, count_seed=0, graph=True, stats=False, host=False, mesh=0,
             constants="scene")


def _case(**kw):
    return {**_STEP, **kw}


def listed():
    return [
        # the smallest call of a program that keeps its particles on the host (a test scene, a tool)
        _case(name="step_block512_host", nx=8, ny=8, nz=8, jitter=0.02, stats=True, graph=False, host=True),
        # the reference's own default scene: 720 particles, its constants, 12 iterations
        _case(name="step_default720", nx=12, ny=5, nz=12, h=0.3, iters=12, stats=True, constants="default"),
        # the configured 4,096-particle block: an interactive simulation, step by step
        _case(name="step_block4096", jitter=0.02, stats=True),
        # a pour onto a triangle mesh (a height field of 2,048 triangles) in mid-motion: odd sizes, more neighbours
        _case(name="step_pour33k_mesh", nx=37, ny=29, nz=31, h=0.05, ratio=2.4, jitter=0.2, speed=0.5, graph=False,
              mesh=32),
        # the configured dam break, as a simulation runs it: graph replay, statistics on
        _case(name="step_dam262k", nx=64, ny=64, nz=64, h=0.025, stats=True),
        # the headline scene: two colliding blocks, 1,048,576 particles
        _case(name="step_blocks1m", nx=64, ny=128, nz=64, h=0.0125, blocks=2),
        # the same through host buffers, as a caller of the C ABI keeps its particles
        _case(name="step_blocks1m_host", nx=64, ny=128, nz=64, h=0.0125, blocks=2, host=True),
        # the configured batch: 256 independent scenes of 2k to 32k particles, 2.8M in all
        _case(name="batch_256scenes", scenes=256, lo=2048, hi=32768, count_seed=4, h=0.05, speed=0.5),
        # the gradient workload: forward with checkpoints and backward through the autograd function
        _case(name="rollout_32k", kind="rollout", nx=32, ny=32, nz=32, h=0.05),
        # one recorded step and its reverse on a large scene
        _case(name="adjoint_262k", kind="adjoint", nx=64, ny=64, nz=64, h=0.025, speed=0.2),
        # the surface of the headline scene over its box, as a viewer or an exporter takes it
        {"name": "surface_blocks1m", **_SURF, "blocks": 2, "nx": 64, "ny": 128, "nz": 64, "h": 0.0125},
        # a frame of it
        {"name": "render_blocks1m", **_REND, "blocks": 2, "nx": 64, "ny": 128, "nz": 64, "h": 0.0125},
    ]


_SURF = dict(kind="surface", nx=32, ny=32, nz=32, h=0.05, ratio=2.0, jitter=0.008, speed=0.0, blocks=1)
_REND = dict(kind="render", nx=32, ny=32, nz=32, h=0.05, ratio=2.0, jitter=0.008, speed=0.0, blocks=1, width=1280,
             height=720, aa=16, depth=3, lights=4)


def _dims(rng, lo, hi):
    """Three sides of a block of lo to hi particles (log-uniform), seldom equal or even."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    side = n ** (1.0 / 3.0)
    nx, ny = max(4, round(side * a)), max(4, round(side * b))
    nz = max(4, min(round(n / (nx * ny)), int(hi / (nx * ny))))
    return nx, ny, nz


def draw(rng):
    kind = rng.choice(["step", "step", "step", "batch", "rollout", "adjoint", "surface", "render"])
    big = {"step": 1 << 20, "adjoint": 1 << 18, "rollout": 1 << 16}.get(kind, 1 << 18)
    nx, ny, nz = _dims(rng, 512, big)
    ratio = rng.choice([2.0, 2.0, round(rng.uniform(1.9, 2.5), 3)])
    # the block fills 0.35 to 0.85 of the unit box's longest side
    h = round(ratio * rng.uniform(0.35, 0.85) / max(nx, ny, nz), 5)
    base = dict(nx=nx, ny=ny, nz=nz, h=h, ratio=ratio, jitter=rng.choice([0.008, 0.05, 0.2]),
                speed=rng.choice([0.0, 0.2, 0.5]))
    if kind == "surface":
        return {**_SURF, **base}
    if kind == "render":
        return {**_REND, **base, "width": rng.randint(160, 1280), "height": rng.randint(90, 720),
                "aa": rng.choice([1, 4, 9]), "depth": rng.randint(1, 3), "lights": rng.choice([1, 2, 4])}
    if kind == "batch":
        lo = rng.randint(300, 4000)
        return _case(scenes=rng.randint(3, 200), lo=lo, hi=lo * rng.randint(2, 12), count_seed=rng.randint(1, 1 << 20),
                     h=rng.choice([0.05, 0.04]), jitter=base["jitter"], speed=base["speed"], graph=rng.random() < 0.7,
                     stats=rng.random() < 0.5)
    if kind in ("rollout", "adjoint"):
        return _case(kind=kind, **base, graph=rng.random() < 0.7)
    return _case(**base, iters=rng.choice([2, 4, 4, 8]), scorr_n=rng.choice([4, 4, 3]), graph=rng.random() < 0.7,
                 stats=rng.random() < 0.5, host=rng.random() < 0.3, mesh=rng.choice([0, 0, 0, 16]))


# ---- inputs ---------------------------------------------------------------------------------

def _params(c):
    if c.get("constants") == "default":  # particles.cpp:20-44 of the reference, with its density for this lattice
        return PbfParams(rest_density=scenes.lattice_density(c["h"], scenes.decimal_square(c["h"]), c["h"] / c["ratio"]),
                         flags=_flags(c))
    return scenes.physical_params(c["h"], c["h"] / c["ratio"], iters=c.get("iters", 4), scorr_n=c.get("scorr_n", 4),
                                  flags=_flags(c), max_neighbors=256 if c["ratio"] > 2.0 or c["jitter"] > 0.1 else 128)


def _flags(c):
    return (PBF_FLAG_GRAPH if c.get("graph") else 0) | (PBF_FLAG_STATS if c.get("stats") else 0)


def _counts(c):
    return scenes.batched_counts(c["count_seed"], c["scenes"], c["lo"], c["hi"]) if c.get("scenes") else []


def _particles(c, seed):
    """Positions and velocities, float32 (n, 3), of one seed."""
    rng = np.random.default_rng(seed)
    s = c["h"] / c["ratio"]
    if c.get("scenes"):
        pos, vel = [], []
        for n in _counts(c):
            side = math.ceil(n ** (1.0 / 3.0))
            p = scenes.lattice(side, side, side, s)[:n]
            at = rng.integers(0, 2, 3) * np.array([1.0, 0.0, 1.0]) * (1.0 - side * s)
            pos.append(p + at)
            vel.append(np.broadcast_to(rng.uniform(-c["speed"], c["speed"], 3), p.shape))
        pos, vel = np.concatenate(pos), np.concatenate(vel).copy()
    elif c["blocks"] == 2:  # side by side along x, moving towards each other
        gap = 0.6 if c["nx"] * s <= 0.4 else 0.5
        a = scenes.lattice(c["nx"], c["ny"], c["nz"], s, corner=(0.0, 0.0, 0.3))
        pos = np.concatenate([a, a + np.array([gap, 0.0, 0.0])])
        vel = 0.01 * rng.standard_normal(pos.shape)
        vel[: len(a), 0] += 1.0
        vel[len(a):, 0] -= 1.0
    elif c.get("constants") == "default":  # the place and the lattice of the reference's particle file
        pos = scenes.lattice(c["nx"], c["ny"], c["nz"], s, corner=(-0.975, 0.425, -0.975))
        vel = np.zeros_like(pos)
    else:
        y0 = 0.16 if c.get("mesh") else 0.0
        corner = [0.5 * (1.0 - c["nx"] * s), min(y0, 1.0 - c["ny"] * s), 0.5 * (1.0 - c["nz"] * s)]
        pos = scenes.lattice(c["nx"], c["ny"], c["nz"], s, corner=corner)
        vel = np.zeros_like(pos)
        vel[:, 1] = -2.0 if c.get("mesh") else 0.0
    pos = pos + rng.uniform(-c["jitter"] * s, c["jitter"] * s, pos.shape)
    if c["speed"] and not c.get("scenes"):
        vel = vel + c["speed"] * rng.uniform(-1.0, 1.0, pos.shape)
    return pos.astype(np.float32), vel.astype(np.float32)


def _height_field(m):
    """2 m^2 triangles of a wavy floor over the unit square, normals up."""
    g = np.linspace(0.0, 1.0, m + 1)
    x, z = np.meshgrid(g, g, indexing="ij")
    p = np.stack([x, 0.1 + 0.05 * np.sin(6 * np.pi * x) * np.cos(6 * np.pi * z), z], -1)
    a, b, c, d = p[:-1, :-1], p[1:, :-1], p[1:, 1:], p[:-1, 1:]
    return np.concatenate([np.concatenate([a, d, c], -1).reshape(-1, 9), np.concatenate([a, c, b], -1).reshape(-1, 9)])


def prepare(case, seed):
    c = case
    prm = _params(c)
    x, v = _particles(c, seed)
    counts = _counts(c)
    if counts:
        sim = pbf.Simulator(x, v, prm, counts=counts, boxes=[(prm.box_lo, prm.box_hi)] * len(counts))
    else:
        sim = pbf.Simulator(x, v, prm)
    if c.get("mesh"):
        sim.set_collider_mesh(_height_field(c["mesh"]))
    st = {"case": c, "prm": prm, "sim": sim}
    n = sim.n
    if c["kind"] == "surface":
        st["lo"], st["hi"] = prm.box_lo, prm.box_hi
        return st
    if c["kind"] == "render":
        scene, st["cam"] = render.cornell_box(prm.box_lo, prm.box_hi)
        sim.set_render_scene(scene)
        st["seed"] = int(seed) % (1 << 30) + 1
        return st
    if c.get("host"):  # page-locked buffers, as a caller that exchanges them every step keeps
        for name, a in (("x", x), ("v", v)):
            st[name] = torch.from_numpy(a).pin_memory().numpy()
        st["xo"], st["vo"] = (torch.empty((n, 3), dtype=torch.float32).pin_memory().numpy() for _ in range(2))
        st["ro"] = torch.empty(n, dtype=torch.float32).pin_memory().numpy()
        return st
    st["x"], st["v"] = torch.from_numpy(x).cuda(), torch.from_numpy(v).cuda()
    if c["kind"] == "step":
        st["xo"], st["vo"] = torch.empty_like(st["x"]), torch.empty_like(st["x"])
        st["ro"] = torch.empty(n, dtype=torch.float32, device="cuda")
        return st
    st["gx"], st["gv"] = (torch.from_numpy(a).cuda() for a in _cotangents(c, x, seed))
    if c["kind"] == "rollout":
        st["rho0"] = torch.tensor(prm.rest_density, dtype=torch.float32, device="cuda")
    return st


def _cotangents(c, x, seed):
    """adjoint: the gradients of the outputs; rollout: the target positions and velocities."""
    rng = np.random.default_rng(seed + (1 << 40))
    if c["kind"] == "rollout":
        s = c["h"] / c["ratio"]
        return ((x + 0.2 * s * rng.standard_normal(x.shape)).astype(np.float32),
                (0.1 * rng.standard_normal(x.shape)).astype(np.float32))
    return rng.standard_normal(x.shape).astype(np.float32), rng.standard_normal(x.shape).astype(np.float32)


# ---- a pass ---------------------------------------------------------------------------------

ROLLOUT_STEPS = 2


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def run(st):
    c, sim, prm = st["case"], st["sim"], st["prm"]
    if c["kind"] == "surface":
        xyz, nrm = sim.surface(lo=st["lo"], hi=st["hi"])
        return {"xyz": xyz, "nrm": nrm}
    if c["kind"] == "render":
        out = sim.render(st["cam"], c["width"], c["height"], c["aa"], c["depth"], c["lights"], seed=st["seed"],
                         lo=prm.box_lo, hi=prm.box_hi)
        return {"hdr": out["hdr"], "rgba": out["rgba"]}
    if c["kind"] == "step" and c["host"]:
        lib = pbf.lib()
        rc = lib.pbf_set_state(sim._h, _ptr(st["x"]), _ptr(st["v"]))
        rc |= lib.pbf_step(sim._h, prm.dt, 1)
        rc |= lib.pbf_get_state(sim._h, _ptr(st["xo"]), _ptr(st["vo"]), _ptr(st["ro"]))
        if rc:
            raise RuntimeError(lib.pbf_last_error(sim._h).decode())
        return {"x": st["xo"], "v": st["vo"], "rho": st["ro"]}
    stream = torch.cuda.current_stream().cuda_stream
    if c["kind"] == "step":
        sim.set_state_device(st["x"].data_ptr(), st["v"].data_ptr(), stream)
        sim.step_async(prm.dt, 1)
        sim.get_state_device(st["xo"].data_ptr(), st["vo"].data_ptr(), st["ro"].data_ptr(), stream)
        return {"x": st["xo"], "v": st["vo"], "rho": st["ro"]}
    if c["kind"] == "adjoint":
        gx, gv, xo, vo = (torch.empty_like(st["x"]) for _ in range(4))
        g_rho0 = torch.empty(1, dtype=torch.float64, device="cuda")
        sim.adjoint_step_device(prm.dt, st["x"].data_ptr(), st["v"].data_ptr(), st["gx"].data_ptr(),
                                st["gv"].data_ptr(), gx.data_ptr(), gv.data_ptr(), g_rho0.data_ptr(), xo.data_ptr(),
                                vo.data_ptr(), stream)
        return {"gx": gx, "gv": gv, "g_rho0": g_rho0.float(), "x": xo, "v": vo}
    x0, v0, rho0 = (st[k].detach().requires_grad_() for k in ("x", "v", "rho0"))
    xt, vt = rollout(sim, x0, v0, rho0, ROLLOUT_STEPS)
    loss = (xt - st["gx"]).square().mean() + 0.01 * (vt - st["gv"]).square().mean()
    gx, gv, g_rho0 = torch.autograd.grad(loss, (x0, v0, rho0))
    return {"gx": gx, "gv": gv, "g_rho0": g_rho0, "x": xt.detach(), "v": vt.detach()}


# ---- what a pass cannot do without -----------------------------------------------------------

def _size(c):
    n = sum(_counts(c)) or c["nx"] * c["ny"] * c["nz"] * c["blocks"]
    nbrs = max(1.0, 0.85 * 4.19 * c["ratio"] ** 3 - 1.0)  # particles within h, surface particles have fewer
    return n, nbrs


def work(case):
    c = case
    n, nbrs = _size(c)
    if c["kind"] == "surface":
        step = 0.5 * c["h"]
        corners = (1.0 / step + 2.0) ** 3
        tris = 8.0 * (n ** (2.0 / 3.0)) * (c["ratio"]) ** 2
        return {"bytes": 12.0 * n + 72.0 * tris, "flops": 10.0 * min(corners, 8.0 * n) * nbrs + 30.0 * tris * nbrs}
    if c["kind"] == "render":
        px = c["width"] * c["height"]
        rays = px * c["aa"] * (1.0 + c["lights"]) * 2.0
        return {"bytes": 12.0 * n + 16.0 * px, "flops": 600.0 * rays}
    # per pair: the predicate; density and lambda, delta p per iteration; XSPH and vorticity; confinement
    fwd = 8.0 + 46.0 * c["iters"] + 34.0 + 20.0
    rev = 60.0 + 40.0 + 85.0 * c["iters"]
    if c["kind"] == "step":
        return {"bytes": 52.0 * n, "flops": n * nbrs * fwd}
    if c["kind"] == "adjoint":
        return {"bytes": 96.0 * n, "flops": n * nbrs * (fwd + rev)}
    return {"bytes": 96.0 * n, "flops": ROLLOUT_STEPS * n * nbrs * (2.0 * fwd + rev)}


# ---- the same in 64 bits ---------------------------------------------------------------------

def _pairs(x, h, h2, scene):
    """(i, j) of all ordered pairs within h of each other in the same scene."""
    cell = 1.0001 * h
    k = torch.floor((x - x.min(0).values) / cell).long() + 1
    d = (k.max(0).values + 2).tolist()
    lin = ((scene * d[2] + k[:, 2]) * d[1] + k[:, 1]) * d[0] + k[:, 0]
    keys, order = torch.sort(lin)
    xs = x[order]
    me = torch.arange(len(x), device=x.device)
    out = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            at = keys + (dz * d[1] + dy) * d[0]
            first, last = torch.searchsorted(keys, at - 1), torch.searchsorted(keys, at + 1, right=True)
            cnt = last - first
            i = torch.repeat_interleave(me, cnt)
            j = torch.arange(len(i), device=x.device) - torch.repeat_interleave(cnt.cumsum(0) - cnt - first, cnt)
            r = xs[i] - xs[j]
            keep = ((r * r).sum(1) <= h2) & (i != j)
            out.append((order[i[keep]], order[j[keep]]))
            del r, keep, i, j
    return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])


def _move(p, d, prm, slide):
    """p moved by d against the box: stop at the nearest clip plane or wall, slide once along a
    wall, stay in the clamp box."""
    length = (d * d).sum(1).sqrt()
    tau = torch.ones_like(length)
    clipped = torch.zeros_like(length, dtype=torch.bool)
    safe = torch.where(d == 0, torch.ones_like(d), d)
    for a, value in prm.clip_planes:
        t = (value - p[:, a]) / safe[:, a]
        take = (d[:, a] != 0) & (t > 0) & (t < tau)
        tau = torch.where(take, t, tau)
        clipped = clipped | take

    def nearest(q, e, es, t):
        wall = torch.full_like(length, -1, dtype=torch.long)
        for a in range(3):
            for side, bound in ((0, prm.box_lo[a]), (1, prm.box_hi[a])):
                tt = ((bound - q[:, a]) / es[:, a]).clamp(min=0)
                take = ((e[:, a] > 0) if side else (e[:, a] < 0)) & (tt <= t)
                t = torch.where(take, tt, t)
                wall = torch.where(take, torch.full_like(wall, 2 * a + side), wall)
        return t, wall

    def on_wall(q, wall):
        cols = []
        for a in range(3):
            col = q[:, a]
            for side, bound in ((0, prm.box_lo[a]), (1, prm.box_hi[a])):
                col = torch.where(wall == 2 * a + side, torch.full_like(col, bound), col)
            cols.append(col)
        return torch.stack(cols, 1)

    tau, wall = nearest(p, d, safe, tau)
    stopped = (wall >= 0) | clipped
    q = torch.where(stopped[:, None], on_wall(p + tau[:, None] * d, wall), p + d)
    if slide:
        axis = torch.div(wall, 2, rounding_mode="floor")
        tan = torch.where(axis[:, None] == torch.arange(3, device=p.device)[None], torch.zeros_like(d), d)
        t2 = (tan * tan).sum(1)
        ok = (wall >= 0) & ~clipped & (t2 > 0)
        tl = torch.where(ok, t2, torch.ones_like(t2)).sqrt()
        e = tan / tl[:, None]
        es = torch.where(e == 0, torch.ones_like(e), e)
        s, wall2 = nearest(q, e, es, 0.5 * length * (1 - tau))
        q = torch.where(ok[:, None], on_wall(q + s[:, None] * e, wall2), q)
    lo = torch.tensor(prm.clamp_lo, dtype=p.dtype, device=p.device)
    hi = torch.tensor(prm.clamp_hi, dtype=p.dtype, device=p.device)
    return torch.where((length > 1e-11)[:, None], torch.minimum(torch.maximum(q, lo), hi), p)


def _step64(x, v, rho0, prm, scene):
    """One step in 64 bits, neighbour sets and collisions fixed for its gradient: x', v', rho."""
    h, h2, n = prm.h, prm.h2, len(x)
    poly6, spiky = 1.56668147106 / h ** 9, -3 * 4.774648292756860 / h ** 6
    dq2 = (prm.scorr_dq * h) ** 2
    tis = 1.0 / (poly6 * (h2 - dq2) ** 3)
    g = torch.tensor(prm.gravity, dtype=x.dtype, device=x.device)
    zero = torch.zeros_like(x)
    xs = x + _lifted(_move, x, (v + g * prm.dt) * prm.dt, prm, True)
    i, j = _pairs(xs.detach(), h, h2, scene)

    def sums(val):
        return torch.zeros((n,) + val.shape[1:], dtype=val.dtype, device=val.device).index_add(0, i, val)

    def kernels(xs):
        r = xs[i] - xs[j]
        r2 = (r * r).sum(1)
        q = (h2 - r2).clamp(min=0)
        rl = r2.clamp(min=1e-22).sqrt()
        s = torch.where((rl > 1e-11) & (rl < h), (h - rl) ** 2 / rl, torch.zeros_like(rl))
        return poly6 * q ** 3, spiky * s[:, None] * r

    for _ in range(prm.iters):
        w, gr = kernels(xs)
        rho, sg, g2 = sums(w), sums(gr), sums((gr * gr).sum(1))
        lam = -(rho / rho0 - 1) / ((g2 + (sg * sg).sum(1)) / rho0 ** 2 + prm.epsilon)
        coef = lam[i] + lam[j] - prm.scorr_k * (w * tis) ** prm.scorr_n
        xs = xs + _lifted(_move, xs, sums(coef[:, None] * gr) / rho0, prm, False)
    u = (xs - x) / prm.dt
    w, gr = kernels(xs)
    du = u[j] - u[i]
    rho, om = sums(w), sums(torch.linalg.cross(du, gr))
    vn = u + prm.xsph_c * sums(w[:, None] * du)
    o2 = (om * om).sum(1)
    mag = torch.where(o2 > 0, torch.where(o2 > 0, o2, torch.ones_like(o2)).sqrt(), torch.zeros_like(o2))
    eta = sums(mag[j][:, None] * gr)
    e2 = (eta * eta).sum(1)
    some = e2 > 1e-22
    nh = eta / torch.where(some, e2, torch.ones_like(e2)).sqrt()[:, None]
    vn = vn + torch.where(some[:, None], prm.dt * prm.vort_eps * torch.linalg.cross(nh, om), zero)
    return xs, vn, rho


def _lifted(move, p, d, prm, slide):
    return move(p, d, prm, slide) - p


MOST_PAIRS_FOR_GRADIENTS = 2.0e7


def exact(case, seed):
    c = case
    # a surface or a frame is this library's own triangulation and random numbers; a mesh
    # collider's stops keep a distance that is a matter of 32-bit coordinates
    if c["kind"] in ("surface", "render") or c.get("mesh"):
        return None
    n, nbrs = _size(c)
    if c["kind"] != "step" and n * nbrs > MOST_PAIRS_FOR_GRADIENTS:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    prm = _params(c)
    x32, v32 = _particles(c, seed)
    x, v = (torch.from_numpy(a).to(dev).double() for a in (x32, v32))
    counts = _counts(c)
    scene = torch.repeat_interleave(torch.arange(max(len(counts), 1), device=dev),
                                    torch.tensor(counts or [len(x)], device=dev))
    if c["kind"] == "step":
        xo, vo, ro = _step64(x, v, prm.rest_density, prm, scene)
        return {"x": xo, "v": vo, "rho": ro}
    rho0 = torch.tensor(prm.rest_density, dtype=torch.float64, device=dev)
    a, b = (torch.from_numpy(t).to(dev).double() for t in _cotangents(c, x32, seed))
    leaves = [t.requires_grad_() for t in (x, v, rho0)]
    xt, vt = x, v
    for _ in range(ROLLOUT_STEPS if c["kind"] == "rollout" else 1):
        xt, vt, _ = _step64(xt, vt, rho0, prm, scene)
    if c["kind"] == "rollout":
        loss = (xt - a).square().mean() + 0.01 * (vt - b).square().mean()
    else:
        loss = (xt * a).sum() + (vt * b).sum()
    gx, gv, gr = torch.autograd.grad(loss, leaves)
    gr = gr if c["kind"] == "rollout" else gr.reshape(1)
    return {"gx": gx, "gv": gv, "g_rho0": gr, "x": xt.detach(), "v": vt.detach()}
