"""The framework's work as measurable cases.

Every case goes through the entry points a program calls: the C ABI of
include/fsim.h and include/fsim_render.h and its Python binding
(fluid_simulator_gb300.native).  Seven kinds of call are covered:

  noalloc    fsim_p2g_noalloc on the caller's buffers and stream
  step       an application that owns its particles hands them over, runs one
             whole fsim_step and takes the result (particles, or the renderer's
             records)
  transfer   particles -> grid (sort, P2G, walls, gravity) -> particles (G2P),
             stage by stage
  solve      one pressure solve of the current grid (fsim_solve_current)
  forward    inference of the pressure warm-start network
  train      one training pass of the network: forward, loss, all gradients
  render     one frame of the screen-space renderer

Inputs are made on the GPU from the seed: particle scenes have a wavy free
surface, uniformly scattered particles (8 per fluid cell) in cell order, as a
running simulation leaves them, and a smooth velocity field of about 1 unit/s,
so that a step moves particles by up to about half a cell.
"""
from __future__ import annotations

import ctypes as C
import math

import torch
import torch.nn.functional as F

from fluid_simulator_gb300 import native as N

DEV = "cuda"
TRANSFER = {"pic": N.PIC, "flip": N.FLIP, "apic": N.APIC}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a frame-budgeted host transfers 52k particles on its own stream
        {"name": "noalloc_32_apic", "kind": "noalloc", "nx": 32, "ny": 32, "nz": 32, "fluid": "dam", "transfer": "apic"},
        # the reference's default scene size: 32^3 FLIP dam break, dt 1/120; latency of a whole step
        {"name": "step_32_flip", "kind": "step", "nx": 32, "ny": 32, "nz": 32, "fluid": "dam", "transfer": "flip",
         "obstacles": False, "tol_rel": False, "publish": "particles"},
        # an odd box (no axis a multiple of 4 or of a tile) with a moving sphere, a source and a sink
        {"name": "step_90x61x75_flip", "kind": "step", "nx": 90, "ny": 61, "nz": 75, "fluid": "fill", "transfer": "flip",
         "obstacles": True, "tol_rel": False, "publish": "particles"},
        # the 128^3 dam break in APIC, dt 1/240: the ordinary production step
        {"name": "step_128_apic", "kind": "step", "nx": 128, "ny": 128, "nz": 128, "fluid": "dam", "transfer": "apic",
         "obstacles": False, "tol_rel": False, "publish": "particles"},
        # the benchmark scene: 256^3 half filled, 65M particles, APIC, moving sphere, disc source and
        # sink box, 1e-6 relative residual, the renderer's records taken after the step
        {"name": "step_256_apic", "kind": "step", "nx": 256, "ny": 256, "nz": 256, "fluid": "fill", "transfer": "apic",
         "obstacles": True, "tol_rel": True, "publish": "gfx"},
        # transfers alone: PIC on an odd box
        {"name": "transfer_107x90x66_pic", "kind": "transfer", "nx": 107, "ny": 90, "nz": 66, "fluid": "fill",
         "transfer": "pic"},
        # transfers alone: the large APIC dam break (the transfer the roofline target is stated for)
        {"name": "transfer_256_apic", "kind": "transfer", "nx": 256, "ny": 256, "nz": 256, "fluid": "dam",
         "transfer": "apic"},
        # pressure projection alone on a random-mask problem (porous fluid, most iterations)
        {"name": "solve_72x100x85_mask", "kind": "solve", "nx": 72, "ny": 100, "nz": 85, "fluid": "mask"},
        # pressure projection alone on a 256^3 dam break: time to 1e-6
        {"name": "solve_256_dam", "kind": "solve", "nx": 256, "ny": 256, "nz": 256, "fluid": "dam"},
        # full-grid inference of the warm-start network inside a 128^3 run
        {"name": "forward_128", "kind": "forward", "n": 1, "nx": 128, "ny": 128, "nz": 128},
        # one training pass of the protocol: 8 crops of 64^3
        {"name": "train_8x64", "kind": "train", "n": 8, "nx": 64, "ny": 64, "nz": 64},
        # one 1000 x 1000 frame of 8M particles with the reference GUI's settings
        {"name": "render_1000_8m", "kind": "render", "width": 1000, "height": 1000, "nx": 128, "ny": 128, "nz": 128,
         "fluid": "fill", "bilateral": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, most):
    """Three axes, each within lo..hi (spread over the logarithm), at most `most` cells."""
    while True:
        base = _log(rng, lo, hi)
        ax = [max(lo, min(hi, int(round(base * rng.uniform(0.6, 1.4))))) for _ in range(3)]
        if ax[0] * ax[1] * ax[2] <= most:
            return ax


def draw(rng):
    """One more case of the listed kinds, sizes spread over their ranges."""
    kind = rng.choice(["noalloc", "step", "step", "transfer", "transfer", "solve", "solve", "forward", "train", "render"])
    if kind == "noalloc":
        nx, ny, nz = _box(rng, 16, 120, 180000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": (nz + 3) // 4 * 4, "fluid": rng.choice(["dam", "fill"]),
                "transfer": rng.choice(["pic", "flip", "apic"])}
    if kind == "step":
        nx, ny, nz = _box(rng, 24, 224, 160 ** 3)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "fluid": rng.choice(["dam", "fill"]),
                "transfer": rng.choice(["pic", "flip", "apic"]), "obstacles": rng.random() < 0.5, "tol_rel": rng.random() < 0.5,
                "publish": rng.choice(["particles", "gfx"])}
    if kind == "transfer":
        nx, ny, nz = _box(rng, 24, 256, 200 ** 3)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "fluid": rng.choice(["dam", "fill"]),
                "transfer": rng.choice(["pic", "flip", "apic"])}
    if kind == "solve":
        fluid = rng.choice(["dam", "fill", "mask"])
        nx, ny, nz = _box(rng, 24, 224, (112 if fluid == "mask" else 192) ** 3)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "fluid": fluid}
    if kind == "forward":
        nx, ny, nz = (8 * ((v + 7) // 8) for v in _box(rng, 24, 192, 128 ** 3))
        return {"kind": kind, "n": 1, "nx": nx, "ny": ny, "nz": nz}
    if kind == "train":
        nx, ny, nz = (8 * ((v + 7) // 8) for v in _box(rng, 16, 72, 64 ** 3))
        return {"kind": kind, "n": max(1, min(rng.randint(1, 16), (8 * 64 ** 3) // (nx * ny * nz))), "nx": nx, "ny": ny, "nz": nz}
    nx, ny, nz = _box(rng, 32, 128, 128 ** 3)
    return {"kind": kind, "width": _log(rng, 320, 1600), "height": _log(rng, 240, 1200), "nx": nx, "ny": ny, "nz": nz,
            "fluid": rng.choice(["dam", "fill"]), "bilateral": rng.random() < 0.5}


# ------------------------------------------------------------------ scenes
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _geometry(case):
    """(cells per axis, cell size, box): the longest axis of the box is about one unit."""
    n = (case["nx"], case["ny"], case["nz"])
    res = float(max(n))
    h = 1.0 / float(torch.tensor(res, dtype=torch.float32))
    return n, h, tuple((k + 0.01) * h for k in n), res


def _dt(case):
    return min(1.0 / 120.0, 1.0 / (1.875 * max(case["nx"], case["ny"], case["nz"])))


def _fluid_cells(case, g):
    """Boolean [nx, ny, nz]: interior cells below a wavy surface ("dam": a block against two
    walls, "fill": the lower half), or a thresholded smooth random field ("mask")."""
    n = (case["nx"], case["ny"], case["nz"])
    ax = [(torch.arange(k, device=DEV, dtype=torch.float32) + 0.5) / k for k in n]
    x, y, z = torch.meshgrid(*ax, indexing="ij")
    ph = torch.rand(4, generator=g, device=DEV) * 6.2831853
    wave = torch.sin(6.2831853 * x + ph[0]) * torch.cos(12.566371 * z + ph[1])
    if case["fluid"] == "dam":
        f = torch.maximum((x - 0.03 * torch.sin(6.2831853 * z + ph[2])) / 0.4, (y - 0.05 * wave) / 0.6)
        share = 0.24
    elif case["fluid"] == "fill":
        f, share = y - 0.04 * wave, 0.5
    else:
        f = _smooth(torch.randn(n, generator=g, device=DEV), 6.0 * max(n) / 256.0 + 1.5)
        share = 0.4 + 0.3 * float(torch.rand(1, generator=g, device=DEV))
    # the lowest cells of the level function, a number that does not depend on the seed (but for "mask")
    inner = f[1:-1, 1:-1, 1:-1]
    fl = torch.zeros(inner.numel(), dtype=torch.bool, device=DEV)
    fl[torch.argsort(inner.flatten())[:max(1, int(share * inner.numel()))]] = True
    return F.pad(fl.view(inner.shape), (1, 1, 1, 1, 1, 1))


def _smooth(f, sigma):
    """Periodic Gaussian smoothing, scaled back to unit variance."""
    t = torch.fft.rfftn(f)
    for a, k in enumerate(f.shape):
        w = torch.fft.rfftfreq(k, device=DEV) if a == 2 else torch.fft.fftfreq(k, device=DEV)
        s = [1, 1, 1]
        s[a] = -1
        t = t * torch.exp(-2.0 * (math.pi * sigma * w) ** 2).view(s)
    f = torch.fft.irfftn(t, s=f.shape)
    return f / f.std()


def _particles(case, g):
    """FP32 positions [n, 3], velocities [n, 3] and APIC matrices [n, 9] in cell order."""
    _, h, _, _ = _geometry(case)
    cells = torch.nonzero(_fluid_cells(case, g)).to(torch.float32)
    pos = (cells[:, None, :] + torch.rand((cells.shape[0], 8, 3), generator=g, device=DEV) * 0.998 + 0.001).view(-1, 3)
    del cells
    for a, k in enumerate((case["nx"], case["ny"], case["nz"])):
        pos[:, a].clamp_(1.26, k - 1.26)  # advection keeps particles this far from the walls
    pos.mul_(h)
    vel = torch.zeros_like(pos)
    grad = torch.zeros((pos.shape[0], 9), device=DEV) if case["transfer"] == "apic" else None
    k = torch.randint(-2, 3, (3, 2, 3), generator=g, device=DEV).float() * 6.2831853
    ph = torch.rand((3, 2), generator=g, device=DEV) * 6.2831853
    for a in range(3):
        for m in range(2):
            arg = pos @ k[a, m] + ph[a, m]
            vel[:, a] += 0.6 * torch.sin(arg)
            if grad is not None:
                arg.cos_().mul_(0.6)
                for b in range(3):
                    grad[:, 3 * a + b] += arg * k[a, m, b]
    return pos, vel, grad


def _obstacles(case, seed):
    n, h, box, _ = _geometry(case)
    dt = _dt(case)
    t = 0.1 + 0.05 * (seed % 7)
    x, xp = 0.1 * math.sin(math.pi * t), 0.1 * math.sin(math.pi * (t - dt))
    b = [k * h for k in n]
    r = 0.15 * min(b)
    sph = (b[0] * 0.5 + x * b[0], b[1] * 0.6, b[2] * 0.5)
    return [N.obstacle(N.OBS_SPHERE, sph, r=r, prev_pos=(b[0] * 0.5 + xp * b[0], sph[1], sph[2]),
                       speed=((x - xp) * b[0] / dt, 0.0, 0.0)),
            N.obstacle(N.OBS_DISC_SOURCE, (b[0] * 0.5, b[1] * 0.95, b[2] * 0.5), r=4 * h, spawn_speed=-1.0),
            N.obstacle(N.OBS_BOX_SINK, (4 * h, 4 * h, 4 * h), size=(8 * h, 8 * h, 8 * h))]


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


# ------------------------------------------------------------------ the network's parameters and inputs
_SPEC = [(27, 16, 16), (27, 16, 16), (1, 128, 32), (27, 32, 32), (27, 32, 32), (1, 256, 64), (27, 64, 64), (27, 64, 64),
         (1, 512, 64), (27, 64, 64), (27, 64, 64), (27, 128, 64), (27, 64, 64), (27, 96, 32), (27, 32, 32), (27, 48, 16),
         (27, 16, 16)]


def _net_params(g):
    """Flat FP32 parameters: He weights, small biases, a random head."""
    parts = []
    for l, (taps, cin, cout) in enumerate(_SPEC):
        w = torch.randn((taps, cout, cin), generator=g, device=DEV) * math.sqrt(2.0 / (taps * (4 if l == 0 else cin)))
        if l == 0:
            w[:, :, 4:] = 0.0
        parts += [w.flatten(), 0.05 * torch.randn(cout, generator=g, device=DEV)]
    parts += [0.25 * torch.randn(16, generator=g, device=DEV), 0.1 * torch.randn(1, generator=g, device=DEV)]
    return torch.cat(parts)


def _net_input(case, g):
    """Batches of pressure problems: rhs / rms and one-hot fluid, solid, air; a smooth target; the fluid mask."""
    xs, ts, ms = [], [], []
    n = (case["nx"], case["ny"], case["nz"])
    for _ in range(case["n"]):
        fl = _fluid_cells({**case, "fluid": "mask" if float(torch.rand(1, generator=g, device=DEV)) < 0.5 else "fill"}, g)
        solid = torch.ones(n, dtype=torch.bool, device=DEV)
        solid[1:-1, 1:-1, 1:-1] = False
        rhs = torch.where(fl, _smooth(torch.randn(n, generator=g, device=DEV), 2.0), 0.0)
        rhs = rhs / (rhs.square().sum() / fl.sum().clamp(min=1)).sqrt()
        xs.append(torch.stack([rhs, fl.float(), solid.float(), (~fl & ~solid).float()], -1))
        t = _smooth(torch.randn(n, generator=g, device=DEV), max(n) / 10.0)
        ts.append(torch.where(fl, 3.0 * t, 0.0))
        ms.append(fl.to(torch.uint8))
    return torch.stack(xs).contiguous(), torch.stack(ts).contiguous(), torch.stack(ms).contiguous()


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind in ("forward", "train"):
        net = N.WarmStartNet(seed=1, out_scale=2.0)
        theta = _net_params(g)
        torch.cuda.synchronize()
        net._check(net.lib.fsim_net_set_params(net.net, _p(theta), N.DEVICE), "fsim_net_set_params")
        x, t, m = _net_input(case, g)
        st.update(net=net, x=x, t=t, m=m, grad=torch.empty_like(theta))
        return st
    n, h, box, res = _geometry(case)
    if kind == "noalloc":
        pos, vel, c = _particles(case, g)
        cells = n[0] * n[1] * n[2]
        desc = N.GridDesc()
        desc.dims[:] = list(box)
        desc.resolution = res
        st.update(lib=N.load_library(), desc=desc, n=pos.shape[0], pos=pos.t().contiguous(), vel=vel.t().contiguous(),
                  c=None if c is None else c.t().contiguous(), u=torch.empty((3, cells), device=DEV),
                  flags=torch.empty(cells, dtype=torch.uint8, device=DEV), avg=torch.empty(cells, device=DEV))
        return st
    if kind == "render":
        pos, vel, _ = _particles({**case, "transfer": "flip"}, g)
        # density: close to 8 inside, falling to 0.5 for the outermost tenth, as avgPNum does at the surface
        dens = 8.0 - 7.5 * torch.clamp(torch.rand(pos.shape[0], generator=g, device=DEV) * 10.0 - 9.0, min=0.0)
        parts = torch.cat([pos, vel.norm(dim=1, keepdim=True), dens[:, None]], 1).contiguous()
        s = 1.0 / 40.0
        prm = N.default_render_params(particle_radius=h / 4, smoothing_size=2.4 * s, transparency_blur_size=2.4 * s,
                                      noise_scale=0.956 / s, bilateral_filter=int(case["bilateral"]))
        for l in range(prm.num_lights):
            for k in range(3):
                prm.lights[l].position[k] *= s
                prm.lights[l].power_density[k] *= s * s
        mid = [0.5 * k * h for k in n]
        eye = (mid[0] + 1.4, mid[1] + 1.0, mid[2] + 1.8)
        yaw, pitch = N.look_at_angles(eye, (mid[0], 0.6 * mid[1], mid[2]))
        W, H = case["width"], case["height"]
        cam = N.camera(eye, yaw, pitch, fov=40.0, aspect=W / H, near=0.05, far=20.0)
        st.update(r=N.Renderer(W, H), parts=parts, prm=prm, cam=cam, color=torch.empty((H, W, 4), device=DEV),
                  depth=torch.empty((H, W), device=DEV))
        return st
    rel = kind == "solve" or case.get("tol_rel", False)
    obst = bool(case.get("obstacles", False))
    prm = N.default_params(transfer=TRANSFER[case.get("transfer", "flip")], resolution=res, tol=1e-6,
                           tol_mode=N.TOL_REL_L2 if rel else N.TOL_ABS_MAX, max_iters=2000 if rel else 200, spawning=obst,
                           despawning=obst)
    sim = N.Simulation(res, prm, dims=box)
    assert sim.shape == n, (sim.shape, n)
    st.update(sim=sim, lib=sim.lib, dt=_dt(case))
    if kind == "solve":
        flags, v2 = _solve_grid(case, g)
        st["p"] = torch.empty(n, device=DEV)
        torch.cuda.synchronize()
        for f, t in [(N.F_FLAGS, flags)] + [(N.F_V2X + a, v2[a]) for a in range(3)]:
            sim._check(sim.lib.fsim_set_grid(sim.ctx, f, _p(t), N.DEVICE), "fsim_set_grid")
        return st
    pos, vel, c = _particles(case, g)
    np_ = pos.shape[0]
    st.update(pos=pos, vel=vel, c=c, n=np_)
    room = np_ + (8192 if obst else 0)
    if kind == "step":
        st["obstacles"] = _obstacles(case, seed) if obst else []
        if case["publish"] == "gfx":
            st["gfx"] = torch.zeros((room, 5), device=DEV)
        else:
            st["out"] = [torch.zeros((room, k), device=DEV) if k < 9 or c is not None else None for k in (3, 3, 9)]
    else:
        torch.cuda.synchronize()
        sim._check(sim.lib.fsim_set_particles(sim.ctx, _p(pos), _p(vel), _p(c), np_, N.DEVICE), "fsim_set_particles")
        st["out"] = [None, torch.empty((np_, 3), device=DEV), torch.empty((np_, 9), device=DEV) if c is not None else None]
        st["u"] = torch.empty((3,) + n, device=DEV)
        st["avg"] = torch.empty(n, device=DEV)
        st["flags"] = torch.empty(n, dtype=torch.uint8, device=DEV)
    return st


def _solve_grid(case, g):
    """Cell types (solid walls) and a smooth random face-velocity field that is zero at solid faces."""
    n = (case["nx"], case["ny"], case["nz"])
    flags = torch.full(n, N.SOLID, dtype=torch.uint8, device=DEV)
    flags[1:-1, 1:-1, 1:-1] = N.AIR
    flags[_fluid_cells(case, g)] = N.WATER
    solid = flags == N.SOLID
    v2 = []
    for a in range(3):
        v = _smooth(torch.randn(n, generator=g, device=DEV), 3.0)
        v[solid | torch.roll(solid, -1, a)] = 0.0
        v2.append(v.contiguous())
    return flags, v2


# ------------------------------------------------------------------ run
def run(st):
    return _RUN[st["kind"]](st)


def _run_noalloc(st):
    u = st["u"]
    rc = st["lib"].fsim_p2g_noalloc(C.byref(st["desc"]), TRANSFER[st["case"]["transfer"]], _p(st["pos"]), _p(st["vel"]),
                                    _p(st["c"]), st["n"], _p(u[0]), _p(u[1]), _p(u[2]), _p(st["flags"]), _p(st["avg"]),
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc:
        raise RuntimeError(f"fsim_p2g_noalloc: {rc}")
    return {"u": u, "avg": st["avg"], "flags": st["flags"]}


def _take_particles(st):
    sim, (p, v, c) = st["sim"], st["out"]
    got = C.c_int64()
    sim._check(sim.lib.fsim_get_particles(sim.ctx, _p(p), _p(v), _p(c), v.shape[0], C.byref(got), N.DEVICE),
               "fsim_get_particles")
    return {"n": got.value, **{k: t for k, t in (("pos", p), ("vel", v), ("c", c)) if t is not None}}


def _run_step(st):
    sim, lib = st["sim"], st["lib"]
    sim._check(lib.fsim_set_particles(sim.ctx, _p(st["pos"]), _p(st["vel"]), _p(st["c"]), st["n"], N.DEVICE),
               "fsim_set_particles")
    sim.set_obstacles(st["obstacles"])
    sim.step(st["dt"])
    if "gfx" not in st:
        return _take_particles(st)
    got = C.c_int64()
    sim._check(lib.fsim_fill_gfx(sim.ctx, C.cast(_p(st["gfx"]), C.POINTER(N.ParticleGfx)), st["gfx"].shape[0], C.byref(got),
                                 N.DEVICE), "fsim_fill_gfx")
    return {"n": got.value, "gfx": st["gfx"]}


def _run_transfer(st):
    sim, dt = st["sim"], st["dt"]
    for stage in (N.STAGE_P2G, N.STAGE_WALLS, N.STAGE_POST_P2G):
        sim.stage(stage, dt)
    for f, t in ((N.F_VX, st["u"][0]), (N.F_VY, st["u"][1]), (N.F_VZ, st["u"][2]), (N.F_AVGPNUM, st["avg"]),
                 (N.F_FLAGS, st["flags"])):
        sim._check(sim.lib.fsim_get_grid(sim.ctx, f, _p(t), N.DEVICE), "fsim_get_grid")
    sim.stage(N.STAGE_G2P, dt)
    return {"u": st["u"], "avg": st["avg"], "flags": st["flags"], **_take_particles(st)}


def _run_solve(st):
    sim = st["sim"]
    sim.solve_current(st["dt"], N.WARM_ZERO)
    sim._check(sim.lib.fsim_get_grid(sim.ctx, N.F_PRESSURE, _p(st["p"]), N.DEVICE), "fsim_get_grid")
    return {"p": st["p"]}


def _run_forward(st):
    return {"out": st["net"].forward(st["x"])}


def _run_train(st):
    net = st["net"]
    out = net.forward(st["x"], train=True)
    net.zero_grad()
    loss = net.backward(st["t"], st["m"])
    net._check(net.lib.fsim_net_get_params(net.net, _p(st["grad"]), 1, N.DEVICE), "fsim_net_get_params")
    return {"out": out, "loss": torch.tensor(loss), "grad": st["grad"]}


def _run_render(st):
    r = st["r"]
    r.frame(st["parts"], st["cam"], st["prm"])
    for img, t in ((N.IMG_COLOR, st["color"]), (N.IMG_DEPTH, st["depth"])):
        r._check(r.lib.fsim_render_read(r.r, img, _p(t), N.DEVICE), "fsim_render_read")
    return {"color": st["color"], "depth": st["depth"]}


_RUN = {"noalloc": _run_noalloc, "step": _run_step, "transfer": _run_transfer, "solve": _run_solve, "forward": _run_forward,
        "train": _run_train, "render": _run_render}


# ------------------------------------------------------------------ work
def work(case):
    """Inputs read once, outputs written once; floating-point operations of the path's formulas
    (a trilinear value or scatter is 8 weights of 3 products per axis; one multigrid-preconditioned
    iteration about 200 operations per fluid cell, about 15 iterations to 1e-6)."""
    kind = case["kind"]
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind in ("forward", "train"):
        vox = cells * case["n"]
        lev = [0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 3, 2, 2, 1, 1, 0, 0]
        flops = sum(2 * t * ci * co * vox / 8 ** l for (t, ci, co), l in zip(_SPEC, lev))
        params = sum(t * ci * co + co for t, ci, co in _SPEC) + 17
        if kind == "forward":
            return {"bytes": vox * 20 + params * 4, "flops": flops}
        return {"bytes": vox * (16 + 4 + 4 + 1) + params * 8, "flops": 3 * flops}
    share = {"dam": 0.24, "fill": 0.5, "mask": 0.55}[case["fluid"]]
    n = 8 * share * cells
    if kind == "render":
        px = case["width"] * case["height"]
        return {"bytes": 20 * n + 20 * px, "flops": 200 * n + 2000 * px}
    if kind == "solve":
        return {"bytes": cells * (1 + 12 + 4), "flops": 3000 * share * cells}
    apic = case["transfer"] == "apic"
    state = 60 if apic else 24
    if kind == "noalloc":
        return {"bytes": state * n + 17 * cells, "flops": (300 if apic else 150) * n}
    if kind == "transfer":
        return {"bytes": state * n + (48 if apic else 12) * n + 17 * cells, "flops": (600 if apic else 300) * n}
    out = 20 if case["publish"] == "gfx" else state
    return {"bytes": (state + out) * n, "flops": (650 if apic else 350) * n + 3000 * share * cells}


# ------------------------------------------------------------------ exact: the same in 64 bits
def exact(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    if kind == "noalloc":
        pos, vel, c = _particles(case, g)
        u, avg, count = _p2g64(case, pos, vel, c)
        return {"u": u.reshape(3, -1), "avg": avg.flatten(), "flags": None}
    if kind == "transfer":
        pos, vel, c = _particles(case, g)
        return _transfer64(case, pos, vel, c)
    if kind == "solve":
        return _solve64(case, *_solve_grid(case, g))
    if kind == "forward":
        theta = _net_params(g).double()
        x, _, _ = _net_input(case, g)
        with torch.no_grad():
            return {"out": _net64(theta, x.double())}
    if kind == "train":
        theta = _net_params(g).double().requires_grad_(True)
        x, t, m = _net_input(case, g)
        out, loss = _loss64(theta, x.double(), t.double(), m.double())
        loss.backward()
        return {"out": out.detach(), "loss": loss.detach(), "grad": theta.grad}
    return None  # a whole step and a frame: no closed form to compare with


def _p2g64(case, pos, vel, c):
    """Trilinear scatter to faces (value = v + C (face - x), normalised where the weight exceeds 1e-6)
    and to cell centres."""
    n, h, _, _ = _geometry(case)
    cells = n[0] * n[1] * n[2]
    u = torch.zeros((3, cells), dtype=torch.float64, device=DEV)
    w = torch.zeros_like(u)
    avg = torch.zeros(cells, dtype=torch.float64, device=DEV)
    count = torch.zeros(cells, dtype=torch.int64, device=DEV)
    for q in range(0, pos.shape[0], 1 << 21):
        p64, v64 = pos[q:q + (1 << 21)].double(), vel[q:q + (1 << 21)].double()
        c64 = None if c is None else c[q:q + (1 << 21)].double()
        gp = p64 / h
        cell = _cells32(case, pos[q:q + (1 << 21)])
        count += torch.bincount(cell, minlength=cells)
        for a in range(4):  # three face fields, then the cell centres
            off = torch.tensor([0.0 if d == a else 0.5 for d in range(3)], device=DEV, dtype=torch.float64)
            base = torch.floor(gp - off)
            f = gp - off - base
            base = base.long()
            for o in range(8):
                b = torch.tensor([(o >> 2) & 1, (o >> 1) & 1, o & 1], device=DEV)
                node = base + b
                wt = torch.where(b.bool(), f, 1.0 - f).prod(1)
                at = node - torch.tensor([1 if d == a else 0 for d in range(3)], device=DEV)  # face k + 1 belongs to cell k
                ok = ((at >= 0) & (at < torch.tensor(n, device=DEV))).all(1)
                wt = torch.where(ok, wt, 0.0)
                idx = ((at[:, 0] * n[1] + at[:, 1]) * n[2] + at[:, 2]).clamp(0, cells - 1)
                if a == 3:
                    avg.index_add_(0, idx, wt)
                    continue
                val = v64[:, a]
                if c64 is not None:
                    val = val + (c64[:, 3 * a:3 * a + 3] * ((node + off) * h - p64)).sum(1)
                w[a].index_add_(0, idx, wt)
                u[a].index_add_(0, idx, wt * val)
    u = torch.where(w > 1e-6, u / w.clamp(min=1e-300), 0.0)
    return u.view(3, *n), avg.view(n), count.view(n)


def _cells32(case, pos):
    """Cell index of each particle (FP32 product, truncated)."""
    n, _, _, res = _geometry(case)
    hinv = torch.tensor(1.0 / (1.0 / float(torch.tensor(res, dtype=torch.float32))), dtype=torch.float32)
    k = (pos * hinv.to(DEV)).long()
    return (k[:, 0] * n[1] + k[:, 1]) * n[2] + k[:, 2]


def _transfer64(case, pos, vel, c):
    n, h, _, _ = _geometry(case)
    u, avg, count = _p2g64(case, pos, vel, c)
    border = torch.ones(n, dtype=torch.bool, device=DEV)
    border[1:-1, 1:-1, 1:-1] = False
    water = (count > 0) & ~border
    for a in range(3):  # a face between a wall cell and a fluid cell does not move
        up = lambda t: t.narrow(a, 1, n[a] - 1)  # noqa: E731
        lo = lambda t: t.narrow(a, 0, n[a] - 1)  # noqa: E731
        stop = (lo(border) & up(water)) | (up(border) & lo(water))
        u[a].narrow(a, 0, n[a] - 1)[stop] = 0.0
    v2 = u.clone()
    free = ~border[:, :-1] & ~border[:, 1:]
    v2[1][:, :-1][free] += -9.81 * _dt(case)
    order = torch.sort(_cells32(case, pos), stable=True)[1]
    pos, vel = pos[order], vel[order]
    flip = case["transfer"] == "flip"
    fr = float(torch.tensor(0.95, dtype=torch.float32)) if flip else 0.0
    out_v = torch.empty(pos.shape, dtype=torch.float64, device=DEV)
    out_c = torch.empty((pos.shape[0], 9), dtype=torch.float64, device=DEV) if c is not None else None
    v2f, uf = v2.view(3, -1), u.view(3, -1)
    for q in range(0, pos.shape[0], 1 << 21):
        s = slice(q, q + (1 << 21))
        gp = pos[s].double() / h
        for a in range(3):
            off = torch.tensor([0.0 if d == a else 0.5 for d in range(3)], device=DEV, dtype=torch.float64)
            base = torch.floor(gp - off)
            f = gp - off - base
            base = base.long()
            val = torch.zeros(gp.shape[0], dtype=torch.float64, device=DEV)
            dif = torch.zeros_like(val)
            gr = [torch.zeros_like(val) for _ in range(3)] if out_c is not None else None
            for o in range(8):
                b = [(o >> 2) & 1, (o >> 1) & 1, o & 1]
                wd = [f[:, d] if b[d] else 1.0 - f[:, d] for d in range(3)]
                at = [base[:, d] + b[d] - (1 if d == a else 0) for d in range(3)]
                idx = (at[0] * n[1] + at[1]) * n[2] + at[2]
                x = v2f[a][idx]
                wt = wd[0] * wd[1] * wd[2]
                val += wt * x
                if flip:
                    dif += wt * (x - uf[a][idx])
                if gr is not None:
                    for d in range(3):
                        sign = torch.where(f[:, d] - b[d] > 0, -1.0, 1.0)
                        e = [k for k in range(3) if k != d]
                        gr[d] += sign / h * wd[e[0]] * wd[e[1]] * x
            out_v[s, a] = val * (1.0 - fr) + (dif + vel[s, a].double()) * fr if flip else val
            if gr is not None:
                for d in range(3):
                    out_c[s, 3 * a + d] = gr[d]
    r = {"u": u, "avg": avg, "flags": None, "vel": out_v}
    if out_c is not None:
        r["c"] = out_c
    return r


def _solve64(case, flags, v2):
    """Conjugate gradients with a diagonal preconditioner to 1e-11 relative residual."""
    n, h, _, _ = _geometry(case)
    fl = flags == N.WATER
    m = fl.double()
    free = (flags != N.SOLID).double()
    v = [t.double() for t in v2]
    sh = lambda t, a, o: torch.roll(t, -o, a)  # noqa: E731  (walls are solid: nothing wraps into the fluid)
    div = sum(v[a] - sh(v[a], a, -1) for a in range(3))
    scale = _dt(case) / (h * h)
    b = -div / h / scale * m
    ns = sum(sh(free, a, o) for a in range(3) for o in (1, -1))
    inv = torch.where(fl, 1.0 / ns.clamp(min=1.0), 0.0)

    def apply(p):
        q = ns * p
        for a in range(3):
            q -= sh(p, a, 1)
            q -= sh(p, a, -1)
        return q.mul_(m)

    x = torch.zeros_like(b)
    r = b.clone()
    z = r * inv
    s = z.clone()
    rz = (r * z).sum()
    bb = float(b.square().sum())
    for it in range(20000):
        q = apply(s)
        alpha = rz / (s * q).sum()
        x.addcmul_(s, alpha.expand_as(s))
        r.addcmul_(q, -alpha.expand_as(q))
        torch.mul(r, inv, out=z)
        rz2 = (r * z).sum()
        s.mul_(rz2 / rz).add_(z)
        rz = rz2
        if it % 100 == 99 and float(r.square().sum()) <= 1e-22 * bb:
            break
    return {"p": x}


class _Layer(torch.autograd.Function):
    """3x3x3 (or pointwise) convolution of [n, d, h, w, c] as shifted matrix products."""

    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        y = None
        for t, sl in _taps(x, w.shape[0]):
            y = sl @ w[t].t() if y is None else y.add_(sl @ w[t].t())
        return y

    @staticmethod
    def backward(ctx, gy):
        x, w = ctx.saved_tensors
        gx = torch.zeros_like(x)
        gw = torch.empty_like(w)
        g2 = gy.reshape(-1, gy.shape[-1])
        for t, sl in _taps(x, w.shape[0]):
            gw[t] = g2.t() @ sl.reshape(-1, sl.shape[-1])
        for t, sl in _taps(gy, w.shape[0]):
            gx += sl @ w[w.shape[0] - 1 - t]
        return gx, gw


def _taps(x, taps):
    if taps == 1:
        yield 0, x
        return
    p = F.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    d, h, w = x.shape[1:4]
    for t in range(27):
        a, b, c = t // 9, t // 3 % 3, t % 3
        yield t, p[:, a:a + d, b:b + h, c:c + w]


def _net64(theta, x):
    at = [0]

    def conv(t):
        taps, cin, cout = _SPEC[conv.l]
        conv.l += 1
        w = theta[at[0]:at[0] + taps * cin * cout].view(taps, cout, cin)
        b = theta[at[0] + taps * cin * cout:at[0] + taps * cin * cout + cout]
        at[0] += taps * cin * cout + cout
        return torch.relu(_Layer.apply(t.contiguous(), w) + b)

    conv.l = 0

    def s2d(t):
        n, d, h, w, c = t.shape
        t = t.view(n, d // 2, 2, h // 2, 2, w // 2, 2, c).permute(0, 1, 3, 5, 2, 4, 6, 7)
        return t.reshape(n, d // 2, h // 2, w // 2, 8 * c)

    def up(t):
        t = F.interpolate(t.permute(0, 4, 1, 2, 3), scale_factor=2, mode="trilinear", align_corners=False)
        return t.permute(0, 2, 3, 4, 1)

    e0 = conv(conv(F.pad(x, (0, 12))))
    e1 = conv(conv(conv(s2d(e0))))
    e2 = conv(conv(conv(s2d(e1))))
    b3 = conv(conv(conv(s2d(e2))))
    d2 = conv(conv(torch.cat([up(b3), e2], -1)))
    d1 = conv(conv(torch.cat([up(d2), e1], -1)))
    d0 = conv(conv(torch.cat([up(d1), e0], -1)))
    return 2.0 * (d0 @ theta[at[0]:at[0] + 16] + theta[at[0] + 16])


def _loss64(theta, x, t, m):
    """Mean over the batch of ||A e|| / ||b|| + 0.1 ||e|| / ||target||, e = out - target on the fluid."""
    out = _net64(theta, x)
    e = (out - t) * m
    free = F.pad(1.0 - x[..., 2], (1, 1, 1, 1, 1, 1))
    pe = F.pad(e, (1, 1, 1, 1, 1, 1))
    d, h, w = e.shape[1:]
    ns, nb = 0.0, 0.0
    for i, j, k in ((2, 1, 1), (0, 1, 1), (1, 2, 1), (1, 0, 1), (1, 1, 2), (1, 1, 0)):
        ns = ns + free[:, i:i + d, j:j + h, k:k + w]
        nb = nb + pe[:, i:i + d, j:j + h, k:k + w]
    r = (ns * e - nb) * m
    norm = lambda v: v.square().sum((1, 2, 3)).sqrt()  # noqa: E731
    return out, (norm(r) / norm(x[..., 0] * m) + 0.1 * norm(e) / norm(t * m)).mean()
