"""Performance cases: the work a simulation has this framework do, each through a public entry point.

Kinds (a case's ``kind``) and what they stand for:

* ``particles``  one step's particle passes through the stage functions an add-on calls: counting sort and
  P2G (``particle_to_grid``), and with ``update`` the G2P / advection pass (``particle_update``) on the
  sorted particles. ``tiled`` is the tolerance mode's P2G, otherwise the reference-order gather.
* ``voxelise``   the collider mesh rasterised into the obstacle mask, as every step with a moving or
  re-voxelised collider does.
* ``solve``      one pressure solve on a prepared ``PressureSolver``: the reference's fixed number of W-cycles
  (``cycles``), a tolerance solve with the default or the tuned preconditioner, and one started from
  the learned warm start with the shipped weights.
* ``step``       a whole ``FlipSolver.step`` of the block scene; the state is put back before each step, so
  every pass does the same work.
* ``batch``      one ``BatchedFlip.step`` of several uneven scenes (state put back likewise).
* ``conv``       one 3-D convolution layer of the warm-start U-Net: the forward pass of inference, or the
  three gradients (weights, bias, input) of a training step.

Cell sizes are powers of two: particle positions in cell units are then exact in float32 and in 64 bits.
"""

from __future__ import annotations

import math

import numpy as np
import torch

DT = 1.0 / 240.0
RHO = 1000.0
NU = 1.0e-6
GRAVITY = (0.0, -9.81, 0.0)
# (input channels, output channels) of the warm-start U-Net's convolutions
LAYERS = [(8, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (48, 16)]


def listed():
    return [
        # config 1 (64^3 dam break, reference semantics): the smallest whole step, bound by launches
        {"name": "step_reference_64", "kind": "step", "nx": 64, "ny": 64, "nz": 64, "fx": 0.4, "fy": 0.6, "fz": 0.4,
         "mode": "reference"},
        # the particle passes of the same scene
        {"name": "particles_reference_64", "kind": "particles", "nx": 64, "ny": 64, "nz": 64, "fx": 0.4, "fy": 0.6,
         "fz": 0.4, "tiled": False, "update": True, "obstacle": False, "flip": 1.0},
        # a domain that is no cube and no multiple of any tile, reference-order P2G only
        {"name": "p2g_reference_odd", "kind": "particles", "nx": 117, "ny": 90, "nz": 139, "fx": 0.9, "fy": 0.5,
         "fz": 0.8, "tiled": False, "update": False, "obstacle": False, "flip": 1.0},
        # the 160^3 block with a collider in the flow, tolerance-mode P2G, FLIP/PIC 0.95
        {"name": "particles_tiled_160", "kind": "particles", "nx": 160, "ny": 160, "nz": 160, "fx": 0.5, "fy": 0.7,
         "fz": 0.5, "tiled": True, "update": True, "obstacle": True, "flip": 0.95},
        # config 2's collider (icosphere of 5120 triangles) voxelised as each of its steps does
        {"name": "voxelise_128", "kind": "voxelise", "n": 128, "subdivisions": 4},
        # the reference's pressure solve: 6 W-cycles from the previous pressure
        {"name": "solve_reference_64", "kind": "solve", "nx": 64, "ny": 64, "nz": 64, "fx": 0.4, "fy": 0.6, "fz": 0.4,
         "cycles": 6, "preset": "default", "learned": False},
        # a tolerance solve with the default options on an odd domain
        {"name": "solve_default_odd", "kind": "solve", "nx": 150, "ny": 104, "nz": 126, "fx": 0.7, "fy": 0.6,
         "fz": 0.9, "cycles": 0, "preset": "default", "learned": False},
        # config 4: the learned warm start at 128^3, tuned preconditioner
        {"name": "solve_learned_128", "kind": "solve", "nx": 128, "ny": 128, "nz": 128, "fx": 1.0, "fy": 0.3,
         "fz": 1.0, "cycles": 0, "preset": "tuned", "learned": True},
        # config 3 and the benchmark's workload: the 256^3 block, ~23M particles, tuned tolerance mode
        {"name": "step_block_256", "kind": "step", "nx": 256, "ny": 256, "nz": 256, "fx": 0.5, "fy": 0.7, "fz": 0.5,
         "mode": "tuned"},
        # config 5 in small: uneven scenes advancing together
        {"name": "batch_6", "kind": "batch", "count": 6, "largest": 96, "pick": 1},
        # the decoder's widest layer at full resolution (inference), and a training batch's layer
        {"name": "conv_forward_128", "kind": "conv", "B": 1, "D": 128, "H": 128, "W": 128, "cin": 48, "cout": 16,
         "backward": False},
        {"name": "conv_backward_8x64", "kind": "conv", "B": 8, "D": 64, "H": 64, "W": 64, "cin": 16, "cout": 16,
         "backward": True},
    ]


def _between(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["particles", "particles", "voxelise", "solve", "solve", "step", "batch", "conv", "conv"])
    grid = {"nx": _between(rng, 24, 176), "ny": _between(rng, 24, 176), "nz": _between(rng, 24, 176),
            "fx": round(rng.uniform(0.35, 1.0), 3), "fy": round(rng.uniform(0.3, 0.75), 3),
            "fz": round(rng.uniform(0.35, 1.0), 3)}
    if kind == "particles":
        return {"kind": kind, **grid, "tiled": rng.random() < 0.5, "update": rng.random() < 0.6,
                "obstacle": rng.random() < 0.4, "flip": rng.choice([1.0, 0.95])}
    if kind == "voxelise":
        return {"kind": kind, "n": _between(rng, 24, 160), "subdivisions": rng.choice([2, 3, 4])}
    if kind == "solve":
        how = rng.choice(["fixed", "default", "tuned", "tuned_fp16", "learned"])
        return {"kind": kind, **grid, "cycles": rng.randint(1, 6) if how == "fixed" else 0,
                "preset": "default" if how in ("fixed", "default") else "tuned_fp16" if how == "tuned_fp16" else "tuned",
                "learned": how == "learned"}
    if kind == "step":
        return {"kind": kind, **grid, "mode": rng.choice(["reference", "tuned"])}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 6), "largest": rng.choice([64, 80, 96]),
                "pick": rng.randrange(1000)}
    cin, cout = rng.choice(LAYERS)
    B, most = rng.randint(1, 8), (1 << 21) * 16 // max(cin, cout)
    D, H = _between(rng, 8, 96), _between(rng, 8, 128)
    W = max(8, min(_between(rng, 8, 160), most // (B * D * H)))
    return {"kind": kind, "B": B, "D": D, "H": H, "W": W, "cin": cin, "cout": cout, "backward": rng.random() < 0.5}


# ---- inputs -----------------------------------------------------------------------------------------
def _generator(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed) * 7919 + 17)


def _shape(case):
    return int(case["nx"]), int(case["ny"]), int(case["nz"])


def _dx(shape):
    return 2.0 ** -math.ceil(math.log2(max(shape)))


def _phases(g):
    return torch.rand(12, generator=g, device="cuda", dtype=torch.float64).tolist()


def _flow(x, y, z, ph, speed=1.0):
    """A smooth velocity field at positions in metres (seeded phases)."""
    t = 2.0 * math.pi
    u = torch.sin(t * (2 * y + ph[0])) * torch.cos(t * (1.5 * z + ph[1])) + 0.3 * torch.sin(t * (5 * x + ph[2]))
    v = torch.sin(t * (2 * z + ph[3])) * torch.cos(t * (1.5 * x + ph[4])) + 0.3 * torch.sin(t * (5 * y + ph[5]))
    w = torch.sin(t * (2 * x + ph[6])) * torch.cos(t * (1.5 * y + ph[7])) + 0.3 * torch.sin(t * (5 * z + ph[8]))
    return speed * u, speed * v, speed * w


def _liquid(case):
    """Boolean mask of the scene's liquid cells (the block, without the ghost layer)."""
    shape = _shape(case)
    axes = [torch.arange(n, device="cuda", dtype=torch.float64) + 0.5 for n in shape]
    inside = [(a > 1) & (a < n - 1) & (a <= f * n) for a, n, f in zip(axes, shape, (case["fx"], case["fy"], case["fz"]))]
    return inside[0][:, None, None] & inside[1][None, :, None] & inside[2][None, None, :]


def _particles(case, seed):
    """Positions and velocities of a running simulation: 8 jittered particles per liquid cell, in the order
    the last step's sort left them, moved one step by a smooth flow with some noise."""
    shape = _shape(case)
    dx = _dx(shape)
    g = _generator(seed)
    ph = _phases(g)
    cells = _liquid(case).nonzero()
    sub = torch.tensor([[a, b, c] for a in (0, 1) for b in (0, 1) for c in (0, 1)], device="cuda", dtype=torch.float32)
    jitter = torch.rand((len(cells), 8, 3), generator=g, device="cuda")
    pos = ((cells[:, None, :].float() + (sub[None] + jitter) * 0.5) * dx).reshape(-1, 3)
    order = torch.argsort(_keys(pos, shape, dx), stable=True)
    pos = pos[order].contiguous()
    vel = torch.stack(_flow(pos[:, 0], pos[:, 1], pos[:, 2], ph), 1)
    vel += 0.05 * torch.randn(vel.shape, generator=g, device="cuda")
    pos = pos + DT * vel
    lo = 1.001 * dx
    for a in range(3):
        pos[:, a].clamp_(np.float32(lo), np.float32((shape[a] - 1.001) * dx))
    return pos.contiguous(), vel.contiguous()


def _keys(pos, shape, dx):
    b = [torch.floor(pos[:, a] * (1.0 / dx) - 0.5).long().clamp_(0, shape[a] - 2) for a in range(3)]
    return (b[0] * shape[1] + b[1]) * shape[2] + b[2]


def _grid_velocity(case, seed):
    """Face velocities of the flow on the grid (u at x faces, v at y faces, w at z faces), float32."""
    shape = _shape(case)
    dx = _dx(shape)
    ph = _phases(_generator(seed + 1000003))
    out = []
    for comp in range(3):
        ax = [(torch.arange(n, device="cuda", dtype=torch.float32) + (1.0 if a == comp else 0.5)) * dx
              for a, n in enumerate(shape)]
        f = _flow(ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :], ph)[comp]
        out.append(f.expand(shape).contiguous())
    return out


def _icosphere(case, seed):
    from continuum_liquid_b200 import scenes

    g = _generator(seed, "cpu")
    r = torch.rand(4, generator=g, dtype=torch.float64).tolist()
    radius = 0.1 + 0.08 * r[0]
    centre = np.array([0.3 + 0.4 * r[1], 0.2 + 0.4 * r[2], 0.3 + 0.4 * r[3]])
    return scenes.icosphere(case.get("subdivisions", 3), radius, centre)


def _sphere_mask(case, seed):
    """Solid cells of a ball in the flow."""
    shape = _shape(case)
    dx = _dx(shape)
    r = torch.rand(3, generator=_generator(seed + 5, "cpu"), dtype=torch.float64).tolist()
    axes = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * dx for n in shape]
    c = [shape[a] * dx * (0.2 + 0.2 * r[a]) for a in range(3)]
    d2 = (axes[0] - c[0])[:, None, None] ** 2 + (axes[1] - c[1])[None, :, None] ** 2 + (axes[2] - c[2])[None, None, :] ** 2
    return (d2 <= (0.12 * min(shape) * dx) ** 2).to(torch.uint8)


def _hydrostatic(case):
    """The previous step's pressure of a block nearly at rest: rho g (surface - y) in the liquid."""
    shape = _shape(case)
    dx = _dx(shape)
    top = case["fy"] * shape[1] * dx
    y = (torch.arange(shape[1], device="cuda", dtype=torch.float32) + 0.5) * dx
    p = (RHO * 9.81 * (top - y)).clamp_min(0.0)[None, :, None].expand(shape)
    return (p * _liquid(case)).contiguous()


def _solve_fields(case, seed):
    """Grid velocity after the forces and the fluid fraction, as the pressure solve meets them."""
    fluid = _liquid(case)
    near = fluid.clone()  # faces of liquid cells: the cell's own and its lower neighbours'
    for a in range(3):
        near |= torch.roll(fluid, -1, a)
    u, v, w = _grid_velocity(case, seed)
    v = v + DT * GRAVITY[1]
    out = []
    for comp, f in enumerate((u, v, w)):
        f = f * near
        f.narrow(comp, 0, 1).zero_()
        f.narrow(comp, f.shape[comp] - 2, 2).zero_()
        out.append(f.contiguous())
    count = torch.randint(5, 12, fluid.shape, generator=_generator(seed + 9), device="cuda").float()
    return out, (fluid * count * 0.125).contiguous()


def _options(preset):
    from continuum_liquid_b200.pressure_solve import TUNED_PRECONDITIONER

    if preset == "default":
        return {}
    return {**TUNED_PRECONDITIONER, "coarse_fp16": preset == "tuned_fp16"}


def prepare(case, seed):
    from continuum_liquid_b200 import batch, learned, particles, pressure_solve, scenes, solver
    from continuum_liquid_b200.backend import default_backend

    k = default_backend()
    kind = case["kind"]
    s = {"case": case, "kernels": k}
    if kind == "particles":
        shape = _shape(case)
        s["pos"], s["vel"] = _particles(case, seed)
        n = len(s["pos"])
        s["n"], s["dx"] = n, _dx(shape)
        s["work"], s["vwork"], s["counts"], s["offsets"], s["sums"] = particles.create_particle_sort_buffers(k, shape, n)
        s["grid"] = [torch.zeros(shape, device="cuda") for _ in range(4)]
        if case["update"]:
            s["new"] = _grid_velocity(case, seed)
            s["obstacle"] = _sphere_mask(case, seed) if case["obstacle"] else None
    elif kind == "voxelise":
        n = case["n"]
        s["tris"] = torch.from_numpy(_icosphere(case, seed)).cuda()
        s["mask"] = torch.zeros((n, n, n), dtype=torch.uint8, device="cuda")
    elif kind == "solve":
        shape = _shape(case)
        s["velocity"], s["ff"] = _solve_fields(case, seed)
        s["previous"] = _hydrostatic(case)
        s["pressure"] = torch.zeros(shape, device="cuda")
        s["solver"] = pressure_solve.PressureSolver(k, shape, _dx(shape), **_options(case["preset"]))
        if case["learned"]:
            net = learned.UNet(k)
            net.load(learned.default_weights_path())
            s["warm"] = learned.LearnedWarmStart(net, shape, _dx(shape))
    elif kind == "step":
        shape = _shape(case)
        s["pos"], s["vel"] = _particles(case, seed)
        s["previous"] = _hydrostatic(case)
        tuned = {"tol": 1e-6, "flip_ratio": 0.95, **_options("tuned")} if case["mode"] == "tuned" else {}
        opts = solver.StepOptions(gravity=GRAVITY, rho=RHO, nu=NU, **tuned)
        s["sim"] = solver.FlipSolver(k, shape, _dx(shape), s["pos"].cpu().numpy(), s["vel"].cpu().numpy(), dt=DT,
                                     options=opts)
    elif kind == "batch":
        sizes = tuple(x for x in (48, 64, 80, 96) if x <= case["largest"])
        several = scenes.uneven_batch(case["count"], seed=case["pick"], sizes=sizes)
        for at, sc in enumerate(several):  # the case's geometry, the seed's particles
            sc.seed = int(seed) * 100 + at
        s["sim"] = batch.BatchedFlip(k, several, tol=1e-6,
                                     **{key: v for key, v in _options("tuned").items() if key != "coarse_fp16"})
        s["pos"], s["vel"] = s["sim"].particles.clone(), s["sim"].particle_velocity.clone()
    else:
        g = _generator(seed)
        vol = (case["B"], case["D"], case["H"], case["W"])
        cin, cout = case["cin"], case["cout"]
        kf, kd = learned.kpad(27 * cin), learned.kpad(27 * cout)
        act = torch.randn((*vol, cin), generator=g, device="cuda").relu_()  # the activations of the layer before
        s["x"] = act.to(torch.bfloat16)
        s["w"] = torch.randn((27 * cin, cout), generator=g, device="cuda") * math.sqrt(2.0 / (27 * cin))
        s["bias"] = 0.1 * torch.randn(cout, generator=g, device="cuda")
        s["wf"] = torch.zeros((cout, kf), dtype=torch.bfloat16, device="cuda")
        s["wd"] = torch.zeros((cin, kd), dtype=torch.bfloat16, device="cuda") if cin >= 16 else None
        k.call("clb_conv3d_arrange_weights", s["w"], s["wf"], s["wd"], cin, cout, kf, kd)
        if case["backward"]:
            s["dy"] = torch.randn((*vol, cout), generator=g, device="cuda").to(torch.bfloat16)
            s["dw"] = torch.zeros((27 * cin, cout), device="cuda")
            s["db"] = torch.zeros(cout, device="cuda")
            s["dx"] = torch.empty_like(s["x"]) if cin >= 16 else None
        else:
            s["y"] = torch.empty((*vol, cout), dtype=torch.bfloat16, device="cuda")
    return s


# ---- one pass ----------------------------------------------------------------------------------------
def run(s):
    from continuum_liquid_b200 import particles, voxelise_mesh

    case, k = s["case"], s["kernels"]
    kind = case["kind"]
    if kind == "particles":
        shape, dx, n = _shape(case), s["dx"], s["n"]
        u, v, w, ff = s["grid"]
        pos, vel, *_ = particles.particle_to_grid(k, None, s["pos"], s["vel"], s["work"], s["vwork"], (u, v, w),
                                                  s["counts"], s["offsets"], s["sums"], ff, n, shape, dx, 8,
                                                  tiled=case["tiled"])
        if case["update"]:
            particles.particle_update(k, None, pos, vel, s["new"], (u, v, w), s["obstacle"], n, shape, dx, DT,
                                      case["flip"], bins=(s["offsets"][0], s["counts"]))
        return {"pos": pos, "vel": vel, "u": u, "v": v, "w": w, "ff": ff, "counts": s["counts"],
                "offsets": s["offsets"][0]}
    if kind == "voxelise":
        n = case["n"]
        s["mask"].zero_()
        voxelise_mesh.voxelise_triangles(k, None, s["tris"], s["mask"], (n, n, n), 1.0 / n, (0.0, 0.0, 0.0))
        return s["mask"]
    if kind == "solve":
        ps, p = s["solver"], s["pressure"]
        p.copy_(s["previous"])
        if case["cycles"]:
            ps.solve(s["velocity"], s["ff"], p, DT, RHO, num_vcycles=case["cycles"])
        else:
            ps.solve(s["velocity"], s["ff"], p, DT, RHO, tol=1e-6, warm_start=s.get("warm"))
        return {"pressure": p, "rhs": ps.rhs}
    if kind == "step":
        sim = s["sim"]
        sim.particles[: sim.n].copy_(s["pos"])
        sim.particle_velocity[: sim.n].copy_(s["vel"])
        sim.pressure.copy_(s["previous"])
        sim.step()
        return {"pos": sim.particles, "vel": sim.particle_velocity, "u": sim.u, "v": sim.v, "w": sim.w,
                "pressure": sim.pressure}
    if kind == "batch":
        sim = s["sim"]
        sim.particles.copy_(s["pos"])
        sim.particle_velocity.copy_(s["vel"])
        sim.pressure.zero_()
        sim.step()
        return {"pos": sim.particles, "vel": sim.particle_velocity, "u": sim.u, "v": sim.v, "w": sim.w,
                "pressure": sim.pressure}
    vol, cin, cout = (case["B"], case["D"], case["H"], case["W"]), case["cin"], case["cout"]
    voxels = math.prod(vol)
    if not case["backward"]:
        k.call("clb_conv3d_forward", s["x"], s["wf"], s["bias"], s["y"], *vol, cin, cout, s["wf"].shape[1], 1)
        return s["y"]
    s["dw"].zero_()
    s["db"].zero_()
    per_block = max(1, (((voxels + 63) // 64) * ((27 * cin + 127) // 128)) // (148 * 8))  # as the network's backward
    k.call("clb_conv3d_wgrad", s["x"], s["dy"], s["dw"], *vol, cin, cout, per_block)
    k.call("clb_unet_bias_grad", s["dy"], s["db"], voxels, cout)
    if s["dx"] is None:  # the first layer's input needs no gradient
        return {"dw": s["dw"], "db": s["db"]}
    k.call("clb_conv3d_dgrad", s["dy"], s["wd"], s["x"], s["dx"], *vol, cout, cin, s["wd"].shape[1])
    return {"dw": s["dw"], "db": s["db"], "dx": s["dx"]}


# ---- what a pass cannot do without ---------------------------------------------------------------------
def _count(case):
    """Particles of a block scene (8 per liquid cell) and cells of its grid."""
    shape = _shape(case)
    liquid = math.prod(max(0, min(int(math.floor(f * n + 0.5)), n - 1) - 1)
                       for n, f in zip(shape, (case["fx"], case["fy"], case["fz"])))
    return 8 * liquid, math.prod(shape)


def work(case):
    kind = case["kind"]
    if kind == "particles":
        n, c = _count(case)
        # particles in and out once; counts, offsets and the four grid fields written; the update reads its grid
        return {"bytes": 48 * n + 24 * c + ((12 * c + (c if case["obstacle"] else 0)) if case["update"] else 0),
                "flops": (250 + (200 if case["update"] else 0)) * n}
    if kind == "voxelise":
        t = 20 * 4 ** case["subdivisions"]
        return {"bytes": case["n"] ** 3 + 36 * t, "flops": 40 * case["n"] ** 3}
    if kind == "solve":
        n, c = _count(case)
        cycles = case["cycles"] or 8
        # velocity, fraction and previous pressure in, rhs and pressure out; one sweep over the liquid a cycle
        return {"bytes": 24 * c + 13 * (n // 8) * cycles, "flops": (60 * cycles) * (n // 8)}
    if kind == "step":
        n, c = _count(case)
        cycles = 1 if case["mode"] == "reference" else 8
        return {"bytes": 48 * n + 40 * c + 13 * (n // 8) * cycles, "flops": 450 * n + 60 * cycles * (n // 8)}
    if kind == "batch":
        cells = case["count"] * (0.7 * case["largest"]) ** 3
        return {"bytes": cells * (0.35 * (48 * 8 + 13 * 8) + 40), "flops": cells * 0.35 * (450 * 8 + 480)}
    v = case["B"] * case["D"] * case["H"] * case["W"]
    cin, cout = case["cin"], case["cout"]
    flops = 54 * cin * cout * v
    if not case["backward"]:
        return {"bytes": 2 * v * (cin + cout) + 54 * cin * cout, "flops": flops}
    dgrad = cin >= 16
    return {"bytes": 2 * v * (cin + cout + (cin if dgrad else 0)) + 4 * 27 * cin * cout,
            "flops": flops * (2 if dgrad else 1)}


# ---- the same in 64 bits -------------------------------------------------------------------------------
def _p2g64(pos, vel, shape, dx):
    """Face velocities and fluid fraction of the sorted particles, in 64 bits."""
    s = pos.double() * (1.0 / dx)
    vel = vel.double()
    cells = math.prod(shape)
    base = [torch.floor(s[:, a] - 0.5).long().clamp_(0, shape[a] - 2) for a in range(3)]
    out = []
    for comp in range(3):
        num = torch.zeros(cells, dtype=torch.float64, device=pos.device)
        den = torch.zeros_like(num)
        spans = [(-1, 0, 1) if a == comp else (0, 1) for a in range(3)]
        for di in spans[0]:
            for dj in spans[1]:
                for dk in spans[2]:
                    wgt, idx, ok = 1.0, 0, True
                    for a, d in enumerate((di, dj, dk)):
                        c = base[a] + d
                        face = c.double() + (1.0 if a == comp else 0.5)
                        wgt = wgt * (1.0 - (s[:, a] - face).abs()).clamp_min(0.0)
                        ok = (c >= 0) & (c < shape[a]) & ok
                        idx = idx * shape[a] + c
                    wgt = wgt * ok
                    idx = idx.clamp_(0, cells - 1)
                    num.index_add_(0, idx, wgt * vel[:, comp])
                    den.index_add_(0, idx, wgt)
        out.append(torch.where(den > 0, num / den.clamp_min(1e-300), torch.zeros_like(num)).view(shape))
    cell = [s[:, a].long().clamp_(1, shape[a] - 2) for a in range(3)]
    count = torch.bincount((cell[0] * shape[1] + cell[1]) * shape[2] + cell[2], minlength=cells)
    return out, (count.double() * 0.125).view(shape)


def _sample64(field, pos, dx, offsets):
    shape = field.shape
    flat = field.reshape(-1)
    base, frac = [], []
    for a in range(3):
        x = pos[:, a] * (1.0 / dx) - offsets[a]
        b = torch.floor(x).long().clamp_(0, shape[a] - 2)
        base.append(b)
        frac.append((x - b).clamp_(0.0, 1.0))
    out = 0.0
    for d in range(8):
        o = (d >> 2, (d >> 1) & 1, d & 1)
        wgt = 1.0
        for a in range(3):
            wgt = wgt * (frac[a] if o[a] else 1.0 - frac[a])
        idx = ((base[0] + o[0]) * shape[1] + base[1] + o[1]) * shape[2] + base[2] + o[2]
        out = out + wgt * flat[idx]
    return out


def _update64(pos, vel, new, old, shape, dx, flip):
    pos, vel = pos.double(), vel.double().clone()
    for comp in range(3):
        off = [1.0 if a == comp else 0.5 for a in range(3)]
        c, o = _sample64(new[comp].double(), pos, dx, off), _sample64(old[comp].double(), pos, dx, off)
        vel[:, comp] = flip * (vel[:, comp] + c - o) + (1.0 - flip) * c
    pos = pos + DT * vel
    for a in range(3):
        lo, hi = 1.001 * dx, (shape[a] - 1.001) * dx
        x = pos[:, a]
        out = (x < lo) | (x > hi)
        y = torch.where(x < lo, 2 * lo - x, x)
        y = torch.where(x > hi, 2 * hi - y, y)
        pos[:, a] = y.clamp(lo, hi)
        vel[:, a] = torch.where(out, torch.zeros_like(x), vel[:, a])
    return pos, vel


def _domain64(vel):
    """Wall faces to zero, the other ghost values from the nearest interior cell."""
    shape = vel[0].shape
    idx = [torch.arange(n, device=vel[0].device).clamp(1, n - 2) for n in shape]
    out = []
    for comp, f in enumerate(vel):
        f = f[idx[0]][:, idx[1]][:, :, idx[2]].clone()
        f.narrow(comp, 0, 1).zero_()
        f.narrow(comp, shape[comp] - 2, 2).zero_()
        out.append(f)
    return out


def _ghost64(p):
    idx = [torch.arange(n, device=p.device).clamp(1, n - 2) for n in p.shape]
    return p[idx[0]][:, idx[1]][:, :, idx[2]]


def _rhs64(vel, fluid, dx):
    b = 0.0
    for a, f in enumerate(vel):
        f = f.double()
        b = b + (f - torch.roll(f, 1, a))
    return (RHO / DT) * (b / dx) * fluid


def _pressure64(b, fluid, dx):
    """laplace(p) = b over the liquid cells (zero pressure in the air, no flow through the walls) by
    Jacobi-preconditioned conjugate gradients, in 64 bits. Worked on the liquid's bounding box."""
    where = fluid.nonzero()
    lo, hi = where.min(0).values.tolist(), where.max(0).values.tolist()
    shape = fluid.shape
    full = torch.zeros(shape, dtype=torch.float64, device=b.device)
    diag = full + 6.0
    for a, n in enumerate(shape):
        diag.narrow(a, 1, 1).sub_(1.0)
        diag.narrow(a, n - 2, 1).sub_(1.0)
    box = tuple(slice(l - 1, h + 2) for l, h in zip(lo, hi))
    inner = (slice(1, -1),) * 3
    m = fluid[box].double()
    diag = diag[box]
    rhs = -(b[box] * (dx * dx)) * m

    def apply(p):
        q = diag * p
        c = q[inner]
        c -= p[2:, 1:-1, 1:-1]
        c -= p[:-2, 1:-1, 1:-1]
        c -= p[1:-1, 2:, 1:-1]
        c -= p[1:-1, :-2, 1:-1]
        c -= p[1:-1, 1:-1, 2:]
        c -= p[1:-1, 1:-1, :-2]
        return q.mul_(m)

    inv = m / diag.clamp_min(1.0)
    x = torch.zeros_like(rhs)
    r = rhs.clone()
    z = inv * r
    d = z.clone()
    rz, stop = (r * z).sum(), 1e-11 * rhs.norm()
    for it in range(6000):
        q = apply(d)
        alpha = rz / (d * q).sum()
        x += alpha * d
        r -= alpha * q
        if it % 20 == 19 and bool(r.norm() <= stop):
            break
        z = inv * r
        new = (r * z).sum()
        d = z + (new / rz) * d
        rz = new
    full[box] = x
    return full


def _step64(pos, vel, shape, dx, flip):
    order = torch.argsort(_keys(pos, shape, dx), stable=True)
    pos, vel = pos[order], vel[order]
    grid, ff = _p2g64(pos, vel, shape, dx)
    old = _domain64(grid)
    fluid = ff > 0
    inside = torch.zeros(shape, dtype=torch.bool, device=pos.device)
    inside[1:-1, 1:-1, 1:-1] = True
    new = []
    for comp, f in enumerate(old):
        lap = sum(torch.roll(f, s, a) for a in range(3) for s in (1, -1)) - 6.0 * f
        new.append(f + DT * GRAVITY[comp] * fluid + NU * DT / (dx * dx) * lap * inside)
    new = _domain64(new)
    p = _ghost64(_pressure64(_rhs64(new, fluid & inside, dx), fluid & inside, dx))
    new = [f - (DT / RHO) * ((torch.roll(p, -1, a) - p) / dx) * inside for a, f in enumerate(new)]
    new = _domain64(new)
    pos, vel = _update64(pos, vel, new, old, shape, dx, flip)
    return {"pos": pos, "vel": vel, "u": new[0], "v": new[1], "w": new[2], "pressure": p}


def _conv64(x, w, sign):
    """sum over taps of x[v + sign * offset(tap)] @ w[tap], zero outside the volume; w: (27, inputs, outputs)."""
    out = torch.zeros((*x.shape[:4], w.shape[2]), dtype=torch.float64, device=x.device)
    n = x.shape[1:4]
    for tap in range(27):
        o = [sign * d for d in (tap // 9 - 1, (tap // 3) % 3 - 1, tap % 3 - 1)]
        dst = tuple(slice(max(0, -d), m - max(0, d)) for d, m in zip(o, n))
        src = tuple(slice(max(0, d), m - max(0, -d)) for d, m in zip(o, n))
        out[(slice(None), *dst)] += x[(slice(None), *src)].double() @ w[tap]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("voxelise", "batch"):  # whole numbers; a whole engine over several scenes
        return None
    if kind == "particles":
        shape = _shape(case)
        dx = _dx(shape)
        pos, vel = _particles(case, seed)
        order = torch.argsort(_keys(pos, shape, dx), stable=True)
        pos, vel = pos[order], vel[order]
        grid, ff = _p2g64(pos, vel, shape, dx)
        p, v = pos.double(), vel.double()
        if case["update"]:
            p, v = (None, None) if case["obstacle"] else _update64(pos, vel, _grid_velocity(case, seed), grid, shape, dx,
                                                                   case["flip"])
        return {"pos": p, "vel": v, "u": grid[0], "v": grid[1], "w": grid[2], "ff": ff, "counts": None, "offsets": None}
    if kind == "solve":
        dx = _dx(_shape(case))
        velocity, ff = _solve_fields(case, seed)
        b = _rhs64(velocity, ff > 0, dx)
        # a fixed number of W-cycles does not reach the solution: its pressure has no such value
        return {"pressure": None if case["cycles"] else _ghost64(_pressure64(b, ff > 0, dx)), "rhs": b}
    if kind == "step":
        if case["mode"] == "reference":
            return None
        pos, vel = _particles(case, seed)
        shape = _shape(case)
        return _step64(pos, vel, shape, _dx(shape), 0.95)
    s = prepare(case, seed)
    cin, cout = case["cin"], case["cout"]
    w = s["w"].to(torch.bfloat16).double().view(27, cin, cout)  # the operands are BF16 by the layer's definition
    x = s["x"].double()
    if not case["backward"]:
        return (_conv64(x, w, 1) + s["bias"].double()).relu_()
    dy = s["dy"].double()
    n = x.shape[1:4]
    dw = torch.zeros((27, cin, cout), dtype=torch.float64, device=x.device)
    for tap in range(27):
        o = (tap // 9 - 1, (tap // 3) % 3 - 1, tap % 3 - 1)
        dst = tuple(slice(max(0, -d), m - max(0, d)) for d, m in zip(o, n))
        src = tuple(slice(max(0, d), m - max(0, -d)) for d, m in zip(o, n))
        dw[tap] = x[(slice(None), *src)].reshape(-1, cin).T @ dy[(slice(None), *dst)].reshape(-1, cout)
    out = {"dw": dw.view(27 * cin, cout), "db": dy.sum((0, 1, 2, 3))}
    if cin >= 16:
        out["dx"] = _conv64(dy, w.transpose(1, 2), -1) * (x > 0)
    return out
