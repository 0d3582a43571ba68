"""Benchmark: FLIP steps/s on the 256^3 block scene (~23M particles) and Poisson ms to 1e-6.

One "step" is one full FLIP timestep of the hot path (binning + counting sort + P2G, grid forces and
boundary conditions, pressure solve to a 1e-6 relative residual by W-cycle preconditioned flexible CG
with FP64 accumulation, projection, fused G2P/advection/particle BCs). Synthetic scene: seeded, see
continuum_liquid_b200/scenes.py.

The "poisson" object compares, on the same systems (the timed run's next steps), the time to a 1e-6
relative residual of: the reference method (FP32 W-cycles on the FP32 pressure, which stalls above
1e-6 at this size: its stall level is reported), W-cycles in FP64 iterative refinement, the flexible
CG, and the flexible CG warm-started by the learned network (when trained weights exist).

  python bench.py [--gpus N --steps K --warmup W]         this backend (value, e2e, roofline, cpu_baseline)
  python bench.py --impl reference [...]                  the reference algorithm on the host cores (the
                                                          CPU restatement; the OpenCL original cannot run here)

Under torchrun with N > 1 every rank advances an independent replica of the scene (the solver is
single-GPU; scenes do not exchange data), the timed region is bracketed by barriers and the time is
the max over ranks.
"""

from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "steps/s at 256^3; Poisson ms to 1e-6 rel. residual, learned vs plain W-cycle"
UNIT = "steps/s"
TOL = 1e-6
COARSE_ITERATION_CHOICES = (64, 16, 8, 4)  # 64: the reference W-cycle's coarsest-level iterations
SMOOTHING_CHOICES = ((2, 4), (2, 2), (1, 2), (1, 1))  # (pre, post); (2, 4): the reference W-cycle's
# factor of every prolonged correction in the W-cycle preconditioner; 1.0: the reference's prolongation
PROLONG_SCALE_CHOICES = (1.0, 1.7)
# the W-cycle preconditioner settings the Poisson comparison picks at 256^3, used by the other cases
TUNED_WCYCLE = {"coarse_iterations": 0, "pre_smooth": 1, "post_smooth": 2, "prolong_scale": 1.8,
                "coarse_smooth": (1, 0)}
SCALED_COARSE_ITERATIONS = (4, 0)  # coarsest-level iterations tried with the larger factors
# (level-0 (pre, post) sweeps, coarse-level (pre, post) sweeps, factor) tried with 0 coarsest-level
# iterations: with the scaled prolongation the coarse levels' post-smoothing can go, and a sweep more on
# level 0 can save a cycle
COARSE_SMOOTH_VARIANTS = (((1, 1), (1, 0), 1.7), ((1, 1), (1, 0), 1.8), ((1, 2), (1, 0), 1.7), ((1, 2), (1, 0), 1.8),
                          ((1, 3), (1, 0), 1.8), ((1, 4), (1, 0), 1.8), ((2, 3), (1, 0), 1.8))
# DRAM bytes (read + write) per launch from one ncu capture of the kernel named (profiles/)
NCU_TRAFFIC_BYTES = {"k_rbgs_colour<true,4>": 95_471_872 + 12_911_360,
                     "k_rbgs_colour_tiles<true,4>": 27_892_224 + 256}
# fluid tiles listed when the tile sweep above was captured (bench.py --case sweep0): its traffic is scaled to
# the tile count of the measured launch (the sweep streams each listed tile and its stencil neighbours)
NCU_TILES_AT_CAPTURE = {"k_rbgs_colour_tiles<true,4>": 5715}
# algorithmic bytes per grid cell of the listed fused level-0 tiles (--case sweep0 --fused-level0): the
# pre-smoothing launch reads b 4 and the
# operator 1, writes x 4 and level 1's p and b (8 per coarse cell = 1 per fine cell); the post-smoothing
# launch reads x 4, the operator 1, b 4 and level 1's p (4 per coarse cell = 0.5 per fine cell), writes x 4
LEVEL0_PRE_BYTES, LEVEL0_POST_BYTES = 10.0, 13.5


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--size", type=int, default=256, help="grid size n of the n^3 block scene")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--method", choices=["fcg", "refine"], default="fcg", help="tolerance-mode pressure iteration")
    ap.add_argument("--learned", choices=["auto", "on", "off"], default="auto",
                    help="learned warm start in the timed steps (auto: when trained weights exist and the Poisson "
                         "comparison shows it faster)")
    ap.add_argument("--poisson-steps", type=int, default=3, help="steps of the Poisson comparison (0: skip)")
    ap.add_argument("--coarse-fp16", choices=["auto", "on", "off"], default="auto",
                    help="FP16 storage of the coarse levels <= 64^3 in the timed steps (auto: when the Poisson "
                         "comparison shows the convergence factor and time hold)")
    ap.add_argument("--coarse-iterations", default="auto",
                    help="red-black iterations of each coarsest-level solve in the W-cycle preconditioner of the timed "
                         "steps (auto: the fastest of 64 (the reference's), 16, 8 and 4 that needs no more FCG cycles "
                         "than 64 in the Poisson comparison)")
    ap.add_argument("--smoothing", default="auto",
                    help="red-black iterations before,after the coarse-grid correction in the W-cycle preconditioner "
                         "of the timed steps, e.g. 2,4 (auto: the fastest of 2,4 (the reference's), 2,2, 1,2 and 1,1 to "
                         "the tolerance in the Poisson comparison, with 4 coarsest-level iterations)")
    ap.add_argument("--prolong-scale", default="auto",
                    help="factor of every correction the W-cycle preconditioner of the timed steps prolongs (1: the "
                         "reference's piecewise-constant prolongation; auto: 1.7 when it is the fastest to the tolerance "
                         "with 4 coarsest-level iterations in the Poisson comparison, together with its smoothing)")
    ap.add_argument("--coarse-smooth", default="auto",
                    help="smoothing sweeps before,after the coarse-grid correction on the levels below the finest in "
                         "the timed steps, e.g. 1,0 (none: the --smoothing counts on every level, the reference; auto: "
                         "the Poisson comparison's choice)")
    ap.add_argument("--single-visit", type=int, default=0,
                    help="first multigrid level visited once (not twice) per visit of the level above in the W-cycle "
                         "preconditioner (0 = the reference's W-cycle; at 256^3 levels 3 and 2 need 20 and 27 FCG "
                         "cycles against 13)")
    ap.add_argument("--case", choices=["step", "sweep0", "wcycle", "batch", "unet", "collider", "particles"],
                    default="step",
                    help="step: the benchmark; sweep0: only level-0 red-black sweeps on the scene's pressure system "
                         "(no particles: a small-memory case for profiling); wcycle: whole W-cycles on that system; "
                         "batch: the batched "
                         "uneven-scenes workload (32 scenes of sizes 48-160, one launch per stage)")
    ap.add_argument("--scenes", type=int, default=32, help="scenes of --case batch")
    ap.add_argument("--sequential-steps", type=int, default=2,
                    help="steps of the one-scene-at-a-time comparison of --case batch (0: skip)")
    ap.add_argument("--sweeps", type=int, default=4,
                    help="red-black iterations (with --fused-level0: launch pairs) of --case sweep0, W-cycles of "
                         "--case wcycle")
    ap.add_argument("--fused-level0", action="store_true",
                    help="--case sweep0/wcycle: level 0 of the W-cycle as the fused tile launches (sweep kind 7)")
    return ap.parse_args()


def batch_case(args):
    """Batched uneven scenes: every scene advances one step per batch step, each pressure solve to TOL."""
    import torch

    from continuum_liquid_b200 import batch, scenes, solver
    from continuum_liquid_b200.backend import Backend

    kernels = Backend(0)
    scs = scenes.uneven_batch(args.scenes, seed=0)
    t0 = time.perf_counter()
    # the W-cycle settings the single-scene comparison picks at 256^3, in the batch and in the
    # one-scene-at-a-time arm alike
    wset = dict(TUNED_WCYCLE)
    b = batch.BatchedFlip(kernels, scs, tol=TOL, **wset)
    setup_s = time.perf_counter() - t0
    for _ in range(args.warmup):
        b.step()
    torch.cuda.synchronize()
    launches0 = kernels.launch_count()
    replays0 = b.graph_replays
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    stats = []
    with ClockSampler(0) as clocks:
        e0.record()
        for _ in range(args.steps):
            stats.append(b.step())
        e1.record()
        torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / args.steps
    line = {
        "case": "batch", "metric": "scene-steps/s of the batched uneven scenes", "unit": "scene-steps/s",
        "value": len(scs) * 1e3 / ms, "ms_per_step": ms, "steps": args.steps, "warmup": args.warmup,
        "config": {"workload": f"uneven_batch_{len(scs)}", "sizes": [s.grid_shape[0] for s in scs],
                   "particles": b.n, "cells": b.C0, "pressure_tolerance": TOL,
                   "pressure_solver": f"per-scene flexible CG preconditioned by one W-cycle (pre {wset['pre_smooth']}, "
                                      f"post {wset['post_smooth']}, coarse {wset['pre_smooth']}+"
                                      f"{wset['coarse_iterations']}, prolonged corrections x{wset['prolong_scale']:g}, "
                                      f"coarser levels {wset.get('coarse_smooth')}), FP64 accumulation"},
        "particles_per_s": b.n * 1e3 / ms,
        "cycles_per_step": [st.cycles for st in stats],
        "rel_residual_max": max(max(st.rel_residual) for st in stats),
        "launches_outside_graphs_per_step": (kernels.launch_count() - launches0) / args.steps,
        "graph_replays_per_step": (b.graph_replays - replays0) / args.steps, "setup_s": setup_s,
        "clocks": clocks.summary(),
    }
    if args.sequential_steps > 0:
        # the same scenes advanced one at a time by the single-scene solver (graphs in its pressure solve)
        del b
        torch.cuda.empty_cache()
        sims = [solver.scene_solver(kernels, sc, solver.StepOptions(flip_ratio=sc.flip_ratio, tol=TOL,
                                                                    gravity=sc.gravity, rho=sc.rho, nu=sc.nu, **wset))
                for sc in scs]
        for sim in sims:
            sim.step()
        torch.cuda.synchronize()
        e0.record()
        for _ in range(args.sequential_steps):
            for sim in sims:
                sim.step()
        e1.record()
        torch.cuda.synchronize()
        seq_ms = e0.elapsed_time(e1) / args.sequential_steps
        line["sequential_single_scene"] = {"ms_per_batch_step": seq_ms, "scene_steps_per_s": len(scs) * 1e3 / seq_ms}
        line["speedup_vs_sequential"] = seq_ms / ms
    print(json.dumps(line), flush=True)


def collider_case(args):
    """The 128^3 collider pool (a falling sphere of liquid into a pool around an icosphere of 5120
    triangles) with the collider voxelised again at every step, each pressure solve to TOL."""
    import torch

    from continuum_liquid_b200 import scenes, solver
    from continuum_liquid_b200.backend import Backend

    kernels = Backend(0)
    sc = scenes.collider_pool(128, seed=0, subdivisions=4)
    opts = solver.StepOptions(flip_ratio=sc.flip_ratio, tol=TOL, gravity=sc.gravity, rho=sc.rho, nu=sc.nu,
                              revoxelise=True, **TUNED_WCYCLE)
    sim = solver.scene_solver(kernels, sc, opts)
    triangles = sum(int(t.shape[0]) for t in sim.colliders)
    for _ in range(args.warmup):
        sim.step()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    stats = []
    with ClockSampler(0) as clocks:
        e0.record()
        for _ in range(args.steps):
            stats.append(sim.step())
        e1.record()
        torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / args.steps
    # the voxelisation alone (brick-culled launch, as in the step), averaged over 20 launches
    e0.record()
    for _ in range(20):
        sim.voxelise_colliders()
    e1.record()
    torch.cuda.synchronize()
    vox_ms = e0.elapsed_time(e1) / 20
    cells = sc.cells
    print(json.dumps({
        "case": "collider", "metric": "steps/s of the 128^3 collider pool, collider voxelised every step",
        "unit": "steps/s", "value": 1e3 / ms, "ms_per_step": ms, "steps": args.steps, "warmup": args.warmup,
        "config": {"workload": "collider_pool_128^3", "grid": list(sc.grid_shape), "particles": sim.n,
                   "triangles": triangles, "pressure_tolerance": TOL, "w_cycle_preconditioner": TUNED_WCYCLE},
        "particles_per_s": sim.n * 1e3 / ms, "cycles_per_step": [s.cycles for s in stats],
        "rel_residual_max": max(s.rel_residual for s in stats),
        "voxelise_ms": vox_ms,
        "voxelise_ray_triangle_tests_per_s_bruteforce_equivalent": cells * triangles / (vox_ms * 1e-3),
        "clocks": clocks.summary()}), flush=True)


def particles_case(args):
    """The particle stages of one step launched alone on the block scene at --size^3 (after one full
    step, so the particles are sorted and moving): count, scan, sort, the reference-order and the tiled
    P2G gather, the fused particle update; device time per launch and algorithmic GB/s. A small-memory
    case for profiling these kernels."""
    import torch

    from continuum_liquid_b200 import scenes, solver
    from continuum_liquid_b200.backend import Backend

    kernels = Backend(0)
    scene = scenes.block(args.size)
    positions, velocities = scenes.seed_particles(scene)
    sim = solver.FlipSolver(kernels, scene.grid_shape, scene.dx, positions, velocities, dt=scene.dt,
                            options=solver.StepOptions(flip_ratio=0.95, tol=TOL, gravity=scene.gravity, rho=scene.rho,
                                                       nu=scene.nu), min_size=scene.min_size)
    for _ in range(max(1, args.warmup)):
        sim.step()
    torch.cuda.synchronize()
    peak, peak_kind = measured_peak_hbm()
    out = {"case": "particles", "grid": list(scene.grid_shape), "particles": sim.n, "peak_gbs": peak,
           "peak_source": peak_kind}
    torch.cuda.nvtx.range_push("stages")
    rows = kernel_rooflines(sim, peak, 1.0, reps=max(1, args.steps))
    sim.options.p2g = "exact"
    rows += [dict(r, stage="p2g_exact") for r in kernel_rooflines(sim, peak, 1.0, reps=max(1, args.steps))
             if r["stage"] == "p2g"]
    torch.cuda.nvtx.range_pop()
    out["stages"] = [{k: r[k] for k in ("stage", "kernels", "ms", "algorithmic_bytes", "achieved", "frac")}
                     for r in rows]
    print(json.dumps(out), flush=True)


def unet_flops_per_voxel() -> float:
    """Convolution FLOPs of one forward pass per full-resolution voxel (2 * 27 * cin * cout per conv
    and voxel of its level; levels 1 and 2 have 1/8 and 1/64 of the voxels)."""
    from continuum_liquid_b200 import learned

    level = {"enc0a": 0, "enc0b": 0, "enc1a": 1, "enc1b": 1, "enc2a": 2, "enc2b": 2, "dec1a": 1, "dec1b": 1,
             "dec0a": 0, "dec0b": 0}
    return sum(2.0 * 27 * cin * cout / 8 ** level[name] for name, cin, cout in learned.LAYERS)


def unet_case(args):
    """U-Net of the learned warm start: forward pass at size^3 and one training step (batch 8 of 64^3
    crops: forward, loss, backward, Adam), device-timed; FLOP rates against the measured BF16 peak."""
    import torch

    from continuum_liquid_b200 import learned
    from continuum_liquid_b200.backend import Backend

    kernels = Backend(0)
    net = learned.UNet(kernels, seed=0)
    fpv = unet_flops_per_voxel()
    peak = None
    path = ROOT / "MEASURED_PEAKS.json"
    if path.exists():
        peak = json.loads(path.read_text()).get("bf16_tflops")
    out = {"case": "unet", "flop_per_voxel_forward": fpv, "peak_bf16_tflops": peak}
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for n in sorted({64, 128, args.size}):
        vol = learned.Vol(1, n, n, n)
        gen = torch.Generator(device="cuda").manual_seed(n)
        net.buffers(vol)["x0"].copy_(torch.randn(vol.voxels, 8, device="cuda", generator=gen).to(torch.bfloat16))
        net.forward(vol)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(3):
            net.forward(vol)
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / 3
        out[f"forward_{n}^3_ms"] = ms
        out[f"forward_{n}^3_tflops"] = fpv * vol.voxels / (ms * 1e-3) / 1e12
        net._buffers.clear()
        torch.cuda.empty_cache()
    vol = learned.Vol(8, 64, 64, 64)
    b = net.buffers(vol)
    gen = torch.Generator(device="cuda").manual_seed(1)
    b["x0"].copy_(torch.randn(vol.voxels, 8, device="cuda", generator=gen).to(torch.bfloat16))
    b["target"].copy_(torch.randn(vol.voxels, device="cuda", generator=gen))
    b["mask"].fill_(1.0)

    def train_step():
        net.forward(vol)
        net.loss_and_grad(vol)
        net.backward(vol)
        net.adam_step(1e-4)

    train_step()
    torch.cuda.synchronize()
    e0.record()
    for _ in range(3):
        train_step()
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / 3
    out["train_step_batch8_64^3_ms"] = ms
    out["train_step_tflops"] = 3.0 * fpv * vol.voxels / (ms * 1e-3) / 1e12  # forward + 2x for the backward
    print(json.dumps(out), flush=True)


def sweep_case(args):
    """Level-0 red-black Gauss-Seidel iterations on the block scene's liquid mask (random right-hand side),
    with the autotuned sweep kind; prints one JSON line with the device time per iteration. With
    --case wcycle: whole W-cycles on the same system instead (one per --sweeps)."""
    import torch

    from continuum_liquid_b200 import scenes
    from continuum_liquid_b200.autotune import tune_hierarchy
    from continuum_liquid_b200.backend import Backend
    from continuum_liquid_b200.pressure_solve import PressureSolver

    kernels = Backend(0)
    scene = scenes.block(args.size)
    centres = [(np.arange(n, dtype=np.float64) + 0.5) * scene.dx for n in scene.grid_shape]
    X, Y, Z = np.meshgrid(*centres, indexing="ij")
    liquid = scene.sources[0].region(X, Y, Z)
    liquid[[0, -1], :, :] = liquid[:, [0, -1], :] = liquid[:, :, [0, -1]] = False
    ff = torch.from_numpy(liquid.astype(np.float32)).cuda()
    del X, Y, Z
    zero = torch.zeros(scene.grid_shape, dtype=torch.float32, device="cuda")
    ps = PressureSolver(kernels, scene.grid_shape, scene.dx, min_size=scene.min_size, autotune=False,
                        coarse_fp16=args.coarse_fp16 == "on")
    ps.prepare((zero, zero, zero), ff, scene.dt, scene.rho)
    gen = torch.Generator(device="cuda").manual_seed(0)
    ps.rhs.copy_(torch.randn(scene.grid_shape, device="cuda", generator=gen) * ff)
    h = ps.hierarchy
    if ps.coarse_fp16:
        h.residual_norms(zero, ps.rhs)  # the FP16 levels' scale comes from the right-hand side's norm
    tune_hierarchy(h, ps.correction, ps.residual)
    kernels.call("clb_mg_set_option", 4, args.single_visit)
    if args.fused_level0:
        h.set_sweep(0, 7)  # level 0 of the W-cycle as the fused tile launches of csrc/mg_level0.cuh
    p = torch.zeros_like(zero)
    h.smooth(0, 2, p, ps.rhs, zero_outside=True)  # p is 0 outside the fluid: the fluid-tile sweep
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    if args.case == "wcycle":
        # as the tolerance mode runs it: a correction from zero (the buffer zeroed once, each W-cycle's
        # first sweep ignoring the previous correction), fluid tiles on every level
        k = 4 if args.coarse_iterations == "auto" else int(args.coarse_iterations)
        pre, post = (2, 4) if args.smoothing == "auto" else (int(x) for x in args.smoothing.split(","))
        w = 1.0 if args.prolong_scale == "auto" else float(args.prolong_scale)
        cs = None if args.coarse_smooth in ("auto", "none") else tuple(int(x) for x in args.coarse_smooth.split(","))
        p.zero_()

        def cycle():
            h.w_cycle(p, ps.rhs, pre_smooth=pre, post_smooth=post, coarse_iterations=k, x_from_zero=True,
                      prolong_scale=w, coarse_smooth=cs)

        cycle()
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_push("sweeps")
        e0.record()
        for _ in range(args.sweeps):
            cycle()
        e1.record()
        torch.cuda.nvtx.range_pop()
        torch.cuda.synchronize()
        print(json.dumps({"case": "wcycle", "grid": list(scene.grid_shape), "levels": [list(x) for x in h.shapes],
                          "sweep_kinds": h.sweeps(), "coarse_iterations": k, "smoothing": [pre, post],
                          "prolong_scale": w, "coarse_smooth": list(cs) if cs else None,
                          "ms_per_w_cycle": e0.elapsed_time(e1) / args.sweeps}), flush=True)
        return
    if not args.fused_level0:
        torch.cuda.nvtx.range_push("sweeps")
        e0.record()
        h.smooth(0, args.sweeps, p, ps.rhs, zero_outside=True)
        e1.record()
        torch.cuda.nvtx.range_pop()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / args.sweeps
        tiles0 = int(h.tile_counts[0].item())
        cells = tiles0 * 4 * (128 if scene.grid_shape[2] % 4 == 0 else 32)
        print(json.dumps({"case": "sweep0", "grid": list(scene.grid_shape), "fluid_tiles": tiles0,
                          "tile_cells": cells, "ms_per_iteration": ms,
                          "algorithmic_gb_s": 13.0 * cells / (ms * 1e-3) / 1e9}), flush=True)
        return
    # the fused level-0 part of a W-cycle: the pre-smoothing launch (from zero, with the restriction) and
    # the post-smoothing launch (with the prolongation), alternating between x and the second buffer
    alt = h.alt[0]

    def pair():
        h.level0_iteration(None, alt, ps.rhs, 3)
        h.level0_iteration(alt, p, ps.rhs, 4)

    pair()
    torch.cuda.synchronize()
    torch.cuda.nvtx.range_push("sweeps")
    e0.record()
    for _ in range(args.sweeps):
        pair()
    e1.record()
    torch.cuda.nvtx.range_pop()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / args.sweeps
    tiles = int(h.fused_tile_count.item())
    cells = h.fused_tile_cells()
    bytes_ = (LEVEL0_PRE_BYTES + LEVEL0_POST_BYTES) * cells
    print(json.dumps({"case": "sweep0", "grid": list(scene.grid_shape), "kernels": "k_l0_iter_tiles<3> + <4>",
                      "fused_tiles": tiles, "tile_cells": cells, "ms_per_pair": ms,
                      "algorithmic_gb_s": bytes_ / (ms * 1e-3) / 1e9}), flush=True)


def workload_config(size, n_particles, args):
    """The workload, identical in both arms' lines (how each arm solves is in its "solver" key)."""
    return {
        "workload": f"flip_step_block_{size}^3",
        "grid": [size, size, size],
        "particles": int(n_particles),
        "liquid_block": [[0, 0, 0], [0.5, 0.7, 0.5]],
        "seeding": "8 particles per liquid cell, one uniform in each 2x2x2 sub-cell, numpy default_rng(0)",
        "dt": 1.0 / 240.0,
        "gravity": [0.0, -9.81, 0.0],
        "flip_ratio": 0.95,
        "pressure_tolerance": TOL,
        "pressure_residual": "FP64 ||b - A p||_2 / ||b||_2 over the interior fluid cells, checked every step",
        "l2": "inputs larger than L2 (particle state 24 B x N, grid fields 4 B x n^3 each)",
        "parallelism": "replicas" if args.gpus > 1 else "single",
    }


def solver_description(method, pre, post, k, fp16_levels=None, single_from=0, prolong_scale=1.0, coarse_smooth=None):
    storage = f", levels {fp16_levels[0][0]}^3 and coarser stored in FP16" if fp16_levels else ""
    if prolong_scale != 1.0:
        storage += f", prolonged corrections x{prolong_scale:g}"
    if coarse_smooth:
        storage += f", coarser levels pre {coarse_smooth[0]}, post {coarse_smooth[1]}"
    cycle = "W-cycle" if not single_from else f"W-cycle (levels {single_from}+ visited once per parent visit)"
    if method == "fcg":
        return (f"flexible CG preconditioned by one {cycle} computed in FP32 (pre {pre}, post {post}, coarse "
                f"{pre}+{k}{storage}), FP64 pressure, residual and norms")
    return (f"{cycle} computed in FP32 (pre {pre}, post {post}, coarse {pre}+{k}{storage}) in FP64 iterative "
            f"refinement")


class ClockSampler:
    """nvidia-smi sampler running during the timed region (clocks and throttle reasons)."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.device_index = device_index
        self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.device_index}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=self.file, stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        self.file.flush()
        rows = []
        with open(self.file.name) as fh:
            for line in fh:
                parts = [p.strip() for p in line.split(",")]
                if len(parts) >= 9:
                    rows.append(parts)
        os.unlink(self.file.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"], "samples": 0}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        sm_max = max((float(r[2]) for r in rows if r[2].replace(".", "").isdigit()), default=None)
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower() == "active"})
        loaded = sorted(sm)[len(sm) // 2:] if sm else []
        return {"sm_mhz": float(np.median(loaded)) if loaded else None, "sm_max_mhz": sm_max, "reasons": reasons,
                "samples": len(rows)}


def measured_peak_hbm():
    path = ROOT / "MEASURED_PEAKS.json"
    if path.exists():
        try:
            return float(json.loads(path.read_text())["hbm_gbs"]), "measured"
        except (KeyError, ValueError):
            pass
    return 6650.0, "fallback"


# ------------------------------------------------------------------------------------------------
# the tolerance-mode preconditioner settings the GPU's Poisson comparison picks at 256^3 (4 coarsest-level
# iterations, one smoothing sweep before and after): the CPU solves to the tolerance with the same iteration
CPU_FCG = {"coarse_iterations": 4, "pre_smooth": 1, "post_smooth": 1}
REFERENCE_FIXED_CYCLES = 6


def cpu_sim(scene, positions, velocities, tol=TOL, cycles=None, **fcg):
    """The reference algorithm on the host cores: the oracle (every reference kernel restated in C++
    with OpenMP, the step order of solver.py:243-529). With ``tol`` each pressure is solved to that
    FP64 relative residual by the flexible CG with the reference's W-cycle as preconditioner (the same
    work as the GPU's timed step); with ``cycles`` by the reference's own method, that fixed number of
    FP32 W-cycles. ``fcg``: preconditioner settings replacing CPU_FCG's (coarse_iterations, pre_smooth,
    post_smooth) or adding prolong_scale and coarse_smooth (the timed steps' choices)."""
    from oracle import oracle

    return oracle.OracleSim(scene.grid_shape, scene.dx, positions, velocities, dt=scene.dt, flip_ratio=0.95,
                            gravity=scene.gravity, rho=scene.rho, nu=scene.nu, min_size=scene.min_size,
                            num_vcycles=cycles or 1, tol=None if cycles else tol, **{**CPU_FCG, **fcg})


def cpu_steps(sim, steps):
    """Seconds and pressure cycles of each of ``steps`` full steps."""
    times, cycles = [], []
    for _ in range(steps):
        t0 = time.perf_counter()
        sim.step()
        times.append(time.perf_counter() - t0)
        cycles.append(int(sim.last_cycles))
    return times, cycles


def cpu_threads():
    from oracle import oracle

    return int(oracle.lib().orc_num_threads())


def reference_method_step(sim):
    """One more step of ``sim`` with the reference's own pressure method (a fixed count of FP32 W-cycles
    from the previous pressure): its time and the FP64 relative residual it leaves."""
    from oracle import oracle

    sim.tol, sim.num_vcycles = None, REFERENCE_FIXED_CYCLES
    t0 = time.perf_counter()
    sim.step()
    sec = time.perf_counter() - t0
    ff = sim.trace["ff"]
    rel = oracle.relative_residual(sim.trace["pressure"], sim.trace["rhs"], ff,
                                   oracle.build_finest_operator(ff, sim.shape), np.float32(sim.dx))
    return {"ms_per_step": sec * 1e3, "w_cycles": REFERENCE_FIXED_CYCLES, "rel_residual": rel,
            "reaches_tolerance": bool(rel <= TOL),
            "method": f"the reference's pressure solve (pressure_solve.py:61-83): {REFERENCE_FIXED_CYCLES} FP32 "
                      f"W-cycles (pre 2, post 4, coarse 2+64) from the previous pressure, no residual check"}


def reference_arm(args):
    """The reference's CPU implementation of the step (the oracle; the OpenCL original needs an OpenCL
    device, which this host lacks) on the same workload, steps and warm-up as this backend's arm."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    from continuum_liquid_b200 import scenes

    scene = scenes.block(args.size)
    positions, velocities = scenes.seed_particles(scene)
    sim = cpu_sim(scene, positions, velocities)
    cpu_steps(sim, args.warmup)
    times, cycles = cpu_steps(sim, args.steps)
    sec = float(np.mean(times))
    value = 1.0 / sec
    threads = cpu_threads()
    fixed = reference_method_step(sim)
    solver = (f"the reference's kernels (oracle restatement, OpenMP) with each pressure solved to {TOL:g} by flexible "
              f"CG preconditioned by the reference W-cycle in FP32 (pre {CPU_FCG['pre_smooth']}, post "
              f"{CPU_FCG['post_smooth']}, coarse {CPU_FCG['pre_smooth']}+{CPU_FCG['coarse_iterations']}), FP64 "
              f"pressure and residual")
    line = {
        "impl": "reference",
        "metric": METRIC,
        "value": value,
        "unit": UNIT,
        "n_gpus": args.gpus,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": sec * 1e3,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic",
        "config": workload_config(args.size, len(positions), args),
        "solver": solver,
        "cycles_per_step": cycles,
        "reference_method": fixed,
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": f"{args.steps} full steps (after {args.warmup} warm-up steps) of the {args.size}^3 "
                                   f"block scene ({len(positions)} particles), each pressure to {TOL:g}"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ------------------------------------------------------------------------------------------------
def load_warm_start(kernels, scene, mode):
    """The learned warm start with the committed trained weights, or (None, reason)."""
    from continuum_liquid_b200 import learned

    path = learned.default_weights_path()
    if mode == "off":
        return None, "disabled"
    if not path.exists():
        if mode == "on":
            raise SystemExit(f"--learned on: no trained weights at {path}")
        return None, f"no trained weights ({path.name} absent)"
    net = learned.UNet(kernels)
    net.load(path)
    return learned.LearnedWarmStart(net, scene.grid_shape, scene.dx), str(path.name)


AUDIT_TOL = 1e-11  # the FP64 reference solution: the same FP64 iteration run this much further


def first_step_parity(sim, positions, velocities, scene):
    """The first step's binning, counting sort and P2G on the GPU (the product path) against the oracle
    on the same seeded particles: per-cell counts, offsets, sorted particles and the P2G grid velocity
    and fluid fraction, compared value for value."""
    from continuum_liquid_b200 import particles as pm
    from oracle import oracle

    k, gs, n = sim.kernels, sim.grid_shape, sim.n
    (sim.particles, sim.particle_velocity, sim.particle_work, sim.particle_velocity_work, _,
     sim.fluid_fraction) = pm.particle_to_grid(k, None, sim.particles, sim.particle_velocity, sim.particle_work,
                                               sim.particle_velocity_work, (sim.u, sim.v, sim.w), sim.bin_counts,
                                               sim.scan_outputs, sim.scan_sums, sim.fluid_fraction, n, gs, sim.dx,
                                               sim.particles_per_cell)
    host = lambda t: t.detach().cpu().numpy()  # noqa: E731
    got = {"counts": host(sim.bin_counts).reshape(gs), "offsets": host(sim.scan_outputs[0]).reshape(gs),
           "sorted_positions": sim.positions(), "sorted_velocities": sim.velocities(), "p2g_u": host(sim.u),
           "p2g_v": host(sim.v), "p2g_w": host(sim.w), "fluid_fraction": host(sim.fluid_fraction)}
    t0 = time.perf_counter()
    pos_s, vel_s, u, v, w, ff, counts, offsets = oracle.particle_to_grid(positions, velocities, scene.dx, gs)
    oracle_s = time.perf_counter() - t0
    ref = {"counts": counts.reshape(gs), "offsets": offsets.reshape(gs), "sorted_positions": pos_s,
           "sorted_velocities": vel_s, "p2g_u": u, "p2g_v": v, "p2g_w": w, "fluid_fraction": ff}
    exact = {name: bool(np.array_equal(got[name], ref[name])) for name in ref}
    return {"scene": f"the first step of the timed scene ({n} particles, {gs[0]}^3)", "bit_exact": exact,
            "all_bit_exact": all(exact.values()), "oracle_s": round(oracle_s, 2),
            "oracle": "CPU restatement of particles.cl:44-227 (pinned to the reference's own bakes by "
                      "tests/test_reference_golden.py)"}


def pressure_error_audit(sim, snapshot, end_positions, steps, min_size):
    """Replays the timed steps from the state they started in, and after each step's pressure solve
    (the timed steps' settings, to TOL) solves the same system once more, in the same FP64 iteration,
    to AUDIT_TOL: the FP64 reference solution. Reports each step's pressure error against it and whether
    the replay reproduced the timed steps bit for bit (the particle positions after the last step)."""
    import torch

    from continuum_liquid_b200.pressure_solve import PressureSolver

    n, pos, vel, pressure = snapshot
    sim.n = n
    sim.particles[:n].copy_(pos)
    sim.particle_velocity[:n].copy_(vel)
    sim.pressure.copy_(pressure)
    ref = PressureSolver(sim.kernels, sim.grid_shape, sim.dx, min_size=min_size, method="fcg", max_cycles=300)
    p_tmp = torch.empty_like(sim.pressure)
    rows = []
    for _ in range(steps):
        p_prev = sim.pressure.clone()
        sim.pre_solve()
        st = sim.solve()
        p_tmp.copy_(p_prev)
        rst = ref.solve((sim.u, sim.v, sim.w), sim.fluid_fraction, p_tmp, sim.dt, sim.options.rho, tol=AUDIT_TOL)
        p, p_star = sim.pressure_solver.pressure64, ref.pressure64
        diff = p - p_star
        rows.append({"cycles": st.cycles, "rel_residual": st.rel_residual,
                     "rel_l2_error": float(torch.linalg.vector_norm(diff) / torch.linalg.vector_norm(p_star)),
                     "rel_max_error": float(diff.abs().max() / p_star.abs().max()),
                     "reference_rel_residual": rst.rel_residual, "reference_cycles": rst.cycles})
        sim.post_solve()
    torch.cuda.synchronize()
    replay_exact = bool(torch.equal(sim.particles[:n], end_positions))
    return {"reference": f"the FP64-accumulated flexible CG run to {AUDIT_TOL:g} on each step's system (FP64 pressure "
                         f"and residual; its FP32 W-cycle preconditioner sets only the convergence rate); checked "
                         f"against the oracle's FP64-only W-cycle solve by tests/test_fp64_reference_gpu.py",
            "steps": rows, "rel_l2_error_max": max(r["rel_l2_error"] for r in rows),
            "rel_max_error_max": max(r["rel_max_error"] for r in rows),
            "replay_bit_exact": replay_exact}


def printed_line(line):
    """The printed line and the parts that go to stderr instead: readers of the line may keep only its last 10,000
    characters, so the per-variant and per-step records are reduced to a time each and to their maxima."""
    poisson, audit = line["poisson"], line["pressure_error"]
    short = dict(line)
    variants = {k: v for k, v in poisson.items() if isinstance(v, dict) and "ms_mean" in v and k != "timed_steps"}
    short["poisson"] = {k: v for k, v in poisson.items() if k not in variants}
    short["poisson"]["variants_ms"] = {k: round(v["ms_mean"], 3) for k, v in variants.items()}
    timed = short["poisson"].get("timed_steps")
    if isinstance(timed, dict):
        short["poisson"]["timed_steps"] = {k: v for k, v in timed.items() if k != "history_last_step"}
    if isinstance(audit, dict):
        short["pressure_error"] = {k: v for k, v in audit.items() if k != "steps"}
    return short, {"poisson": poisson, "pressure_error": audit}


def update_kernel(particles):
    """The particle update a step launches (csrc/g2p_tiled.cuh PUT_MIN_PARTICLES)."""
    return "k_particle_update_tiled" if particles >= 2_300_000 else "k_particle_update"


def p2g_kernel(tiled, cells):
    """The P2G kernel a step launches (csrc/p2g_tiled.cuh P2GT_MIN_CELLS, csrc/p2g_ordered.cuh P2GO_MIN_CELLS)."""
    if tiled and cells >= 3_500_000:
        return "k_p2g_tiled"
    return "k_p2g_ordered" if cells >= 1 << 17 else "k_p2g_gather"


def kernel_rooflines(sim, peak, ms_per_step, reps=5):
    """Device time of each particle stage launched alone (CUDA events on the launching stream, the mean
    of ``reps`` launches on the scene's current state) against its algorithmic bytes."""
    import torch

    from continuum_liquid_b200 import particles as pm

    k, gs, n = sim.kernels, sim.grid_shape, sim.n
    C = int(np.prod(gs))
    scratch = sim.scan_sums[0]
    inv_dx = float(np.float32(1.0 / sim.dx))
    tiled = sim.options.tiled_p2g()
    stages = []

    def timed(name, kernel, bytes_, fn, prepare=None):
        times = []
        for _ in range(reps + 1):
            if prepare is not None:
                prepare()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            fn()
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        ms = float(np.mean(times[1:]))
        gbs = bytes_ / (ms * 1e-3) / 1e9
        stages.append({"stage": name, "kernels": kernel, "ms": ms, "algorithmic_bytes": int(bytes_),
                       "achieved": gbs, "unit": "GB/s", "frac": gbs / peak, "share_of_step": ms / ms_per_step})

    pos, vel = sim.particles, sim.particle_velocity
    timed("count", "k_bin_count", 20 * n + 4 * C,
          lambda: k.call("clb_count_particles_per_cell", pos, sim.bin_counts, scratch.keys, scratch.ranks, n, inv_dx,
                         *gs), prepare=sim.bin_counts.zero_)
    timed("scan", "k_scan_lookback", 8 * C,
          lambda: pm.exclusive_prefix_sum(k, None, sim.bin_counts, sim.scan_outputs, sim.scan_sums, C))
    timed("sort", "k_scatter_perm + k_stable_gather", 56 * n + 4 * C,
          lambda: pm.sort_particles(k, None, pos, vel, sim.particle_work, sim.particle_velocity_work,
                                    sim.scan_outputs[0], sim.bin_counts, scratch, n))
    timed("p2g", p2g_kernel(tiled, C), 24 * n + 24 * C,
          lambda: pm.particle_to_grid_gather(k, None, sim.particle_work, sim.particle_velocity_work,
                                             sim.scan_outputs[0], sim.bin_counts, (sim.u, sim.v, sim.w),
                                             sim.fluid_fraction, gs, sim.dx, sim.particles_per_cell, tiled=tiled))

    # the sort left the particles sorted by bin in the work buffers, with the bins of the scan above: the
    # state the step's particle update runs on
    sorted_pos, sorted_vel = sim.particle_work[:n].clone(), sim.particle_velocity_work[:n].clone()

    def restore():
        sim.particle_work[:n].copy_(sorted_pos)
        sim.particle_velocity_work[:n].copy_(sorted_vel)

    timed("particle_update", f"{update_kernel(n)} (G2P, FLIP/PIC blend, advection, particle BCs)", 48 * n + 24 * C,
          lambda: pm.particle_update(k, None, sim.particle_work, sim.particle_velocity_work, (sim.u, sim.v, sim.w),
                                     (sim.u_work, sim.v_work, sim.w_work), sim.obstacle, n, gs, sim.dx, sim.dt,
                                     sim.options.flip_ratio, bins=(sim.scan_outputs[0], sim.bin_counts)),
          prepare=restore)
    return stages


def poisson_comparison(kernels, sim, steps, warm, min_size):
    """Time to TOL of each pressure iteration on the same systems (the next `steps` steps of `sim`)."""
    import torch

    from continuum_liquid_b200.pressure_solve import PressureSolver

    solvers = {m: PressureSolver(kernels, sim.grid_shape, sim.dx, min_size=min_size, method=m)
               for m in ("refine", "fcg")}
    solvers["fcg_fp16"] = PressureSolver(kernels, sim.grid_shape, sim.dx, min_size=min_size, method="fcg",
                                         coarse_fp16=True)
    # fewer coarsest-level iterations in the W-cycle preconditioner, with either coarse storage
    for k in COARSE_ITERATION_CHOICES[1:]:
        for fp16 in (False, True):
            solvers[f"fcg{'_fp16' if fp16 else ''}_c{k}"] = PressureSolver(
                kernels, sim.grid_shape, sim.dx, min_size=min_size, method="fcg", coarse_fp16=fp16, coarse_iterations=k)
    # fewer smoothing sweeps per level, with 4 coarsest-level iterations and either coarse storage
    for pre, post in SMOOTHING_CHOICES[1:]:
        for fp16 in (False, True):
            solvers[f"fcg{'_fp16' if fp16 else ''}_c4_s{pre}{post}"] = PressureSolver(
                kernels, sim.grid_shape, sim.dx, min_size=min_size, method="fcg", coarse_fp16=fp16, coarse_iterations=4,
                pre_smooth=pre, post_smooth=post)
    # the same with every prolonged correction scaled by each larger factor (names end in _w17 for 1.7),
    # with 4 and with 0 coarsest-level iterations (the scaled W-cycle needs no more cycles without them)
    for name in [n for n in solvers if n.endswith("_c4") or "_c4_s" in n]:
        ps = solvers[name]
        for w in PROLONG_SCALE_CHOICES[1:]:
            for k in SCALED_COARSE_ITERATIONS:
                solvers[f"{name.replace('_c4', f'_c{k}')}_w{round(w * 10)}"] = PressureSolver(
                    kernels, sim.grid_shape, sim.dx, min_size=min_size, method="fcg", coarse_fp16=ps.coarse_fp16,
                    coarse_iterations=k, pre_smooth=ps.pre_smooth, post_smooth=ps.post_smooth, prolong_scale=w)
    for fp16 in (False, True):
        for (pre, post), cs, w in COARSE_SMOOTH_VARIANTS:
            solvers[f"fcg{'_fp16' if fp16 else ''}_c0_s{pre}{post}_w{round(w * 10)}_cs{cs[0]}{cs[1]}"] = \
                PressureSolver(kernels, sim.grid_shape, sim.dx, min_size=min_size, method="fcg", coarse_fp16=fp16,
                               coarse_iterations=0, pre_smooth=pre, post_smooth=post, prolong_scale=w,
                               coarse_smooth=cs)
    single = {}  # variant name -> first level visited once (clb_mg_set_option 4); none by default
    p_tmp = torch.empty_like(sim.pressure)
    rows = {"refine": [], "fcg": [], "fcg_fp16": [], "fcg_learned": [], "fcg_tuned_learned": []}
    rows.update({name: [] for name in solvers if "_c" in name})
    fp32 = []
    rho = sim.options.rho
    for _ in range(steps):
        sim.pre_solve()
        saved = sim.pressure.clone()
        vel = (sim.u, sim.v, sim.w)
        variants = [(name, ps, None) for name, ps in solvers.items()]
        if warm is not None:
            variants.append(("fcg_learned", solvers["fcg"], warm))
            # the same guess with the preconditioner settings the timed steps use (FP16 coarse levels,
            # 4 coarsest-level iterations, one smoothing sweep each way): the comparison that decides
            variants.append(("fcg_tuned_learned", solvers["fcg_fp16_c4_s11"], warm))
        for name, ps, ws in variants:
            kernels.call("clb_mg_set_option", 4, single.get(name, 0))
            for rep in range(2):  # the first run captures graphs and tunes; the second is timed
                p_tmp.copy_(saved)
                st = ps.solve(vel, sim.fluid_fraction, p_tmp, sim.dt, rho, tol=TOL, warm_start=ws, solid=sim.obstacle)
            kernels.call("clb_mg_set_option", 4, 0)
            rows[name].append({"ms": st.device_ms(), "cycles": st.cycles, "rel": st.rel_residual,
                               "guess": st.warm_start, "learned_rel": st.learned_rel_residual,
                               "initial_rel": st.initial_rel_residual,
                               "factor": (st.rel_residual / st.initial_rel_residual) ** (1.0 / st.cycles)
                               if st.cycles and st.initial_rel_residual else None})
        # the reference method: FP32 W-cycles on the FP32 pressure (FP64 residual read after each)
        ps = solvers["refine"]
        p_tmp.copy_(saved)
        ps.solve(vel, sim.fluid_fraction, p_tmp, sim.dt, rho, num_vcycles=0, tol=None)
        h = ps.hierarchy
        hist = [ps.relative_residual(p_tmp)]
        for _ in range(40):
            h.w_cycle(p_tmp, ps.rhs)
            hist.append(ps.relative_residual(p_tmp))
        p_tmp.copy_(saved)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(20):
            h.w_cycle(p_tmp, ps.rhs)
        e1.record()
        torch.cuda.synchronize()
        reached = next((i for i, r in enumerate(hist) if r <= TOL), None)
        fp32.append({"ms_per_cycle": e0.elapsed_time(e1) / 20, "stall_rel": min(hist), "cycles_to_tol": reached})
        sim.solve()
        sim.post_solve()

    def mean(rs, key):
        vals = [r[key] for r in rs if r[key] is not None]
        return float(np.mean(vals)) if vals else None

    out = {"steps": steps, "tolerance": TOL}
    out["fp32_wcycle"] = {
        "reaches_tol": all(f["cycles_to_tol"] is not None for f in fp32),
        "stall_rel_residual": [float("%.3g" % f["stall_rel"]) for f in fp32],
        "ms_per_cycle": float(np.mean([f["ms_per_cycle"] for f in fp32])),
        "note": "FP32 W-cycles on the FP32 pressure (the reference method) over 40 cycles per system; the float32 "
                "rounding of the pressure alone leaves a residual above 1e-6 at this size",
    }
    for name, rs in rows.items():
        if not rs:
            continue
        out[name] = {"ms_mean": mean(rs, "ms"), "cycles_mean": mean(rs, "cycles"),
                     "rel_max": max(r["rel"] for r in rs), "cycles": [r["cycles"] for r in rs],
                     "ms": [round(r["ms"], 3) for r in rs],
                     "convergence_factor_mean": mean(rs, "factor")}
        if name in ("fcg_learned", "fcg_tuned_learned"):
            out[name]["guess_used"] = [r["guess"] for r in rs]
            out[name]["learned_rel"] = [r["learned_rel"] for r in rs]
            out[name]["previous_rel"] = [r["initial_rel"] for r in rows["fcg"]]
    if rows["refine"] and rows["fcg"]:
        out["speedup_fcg_vs_refine"] = out["refine"]["ms_mean"] / out["fcg"]["ms_mean"]
    if rows["fcg_fp16"]:
        f16, f32 = out["fcg_fp16"], out["fcg"]
        f16["fp16_levels"] = [list(sh) for sh in solvers["fcg_fp16"].hierarchy.shapes[
            solvers["fcg_fp16"].hierarchy.fp16_level:]] if solvers["fcg_fp16"].hierarchy.fp16_level else []
        f16["operator_inexact_entries"] = solvers["fcg_fp16"].hierarchy.fp16_inexact_entries()
        # the rule: FP16 coarse storage where the measured convergence factor holds (no more cycles) and it
        # is not slower
        out["coarse_fp16_holds"] = bool(f16["fp16_levels"]) and f16["cycles_mean"] <= f32["cycles_mean"] and \
            f16["ms_mean"] <= f32["ms_mean"] * 1.01
    # the rule for the coarsest-level iterations: with the chosen coarse storage, the fastest count that
    # needs no more cycles than the reference's 64
    base = "fcg_fp16" if out.get("coarse_fp16_holds") else "fcg"
    best_k, best_ms = COARSE_ITERATION_CHOICES[0], out[base]["ms_mean"]
    for k in COARSE_ITERATION_CHOICES[1:]:
        r = out.get(f"{base}_c{k}")
        if r and r["cycles_mean"] <= out[base]["cycles_mean"] and r["ms_mean"] < best_ms:
            best_k, best_ms = k, r["ms_mean"]
    out["coarse_iterations_chosen"] = best_k
    # the rule for the smoothing counts (with 4 coarsest-level iterations chosen): the fastest to the
    # tolerance
    best_s = SMOOTHING_CHOICES[0]
    if best_k == 4:
        best_ms = out[f"{base}_c4"]["ms_mean"]
        for pre, post in SMOOTHING_CHOICES[1:]:
            r = out.get(f"{base}_c4_s{pre}{post}")
            if r and r["ms_mean"] < best_ms:
                best_s, best_ms = (pre, post), r["ms_mean"]
    out["smoothing_chosen"] = list(best_s)
    # the rule for the prolongation factor (with 4 coarsest-level iterations chosen): the fastest to the
    # tolerance of the chosen smoothing with factor 1 and every smoothing and scaled coarsest-level
    # count with a larger factor, which may change the smoothing and the count too
    best_w, best_cs, best_fp16 = PROLONG_SCALE_CHOICES[0], None, base == "fcg_fp16"
    if best_k == 4:
        def c_name(k, s):
            return f"{base}_c{k}" if tuple(s) == SMOOTHING_CHOICES[0] else f"{base}_c{k}_s{s[0]}{s[1]}"

        best_ms = out[c_name(4, best_s)]["ms_mean"]
        for w in PROLONG_SCALE_CHOICES[1:]:
            for k in SCALED_COARSE_ITERATIONS:
                for s in SMOOTHING_CHOICES:
                    r = out.get(f"{c_name(k, s)}_w{round(w * 10)}")
                    if r and r["ms_mean"] < best_ms:
                        best_w, best_k, best_s, best_ms = w, k, s, r["ms_mean"]
        # these variants in either coarse storage: at these settings FP32 and FP16 coarse levels differ
        # by a few per cent, not always in the direction the reference settings showed
        for storage in ("fcg", "fcg_fp16"):
            for s, cs, w in COARSE_SMOOTH_VARIANTS:
                r = out.get(f"{storage}_c0_s{s[0]}{s[1]}_w{round(w * 10)}_cs{cs[0]}{cs[1]}")
                if r and r["ms_mean"] < best_ms:
                    best_w, best_k, best_s, best_cs, best_ms = w, 0, s, cs, r["ms_mean"]
                    best_fp16 = storage == "fcg_fp16"
    out["coarse_fp16_chosen"] = bool(best_fp16)
    out["coarse_smooth_chosen"] = list(best_cs) if best_cs else None
    out["coarse_iterations_chosen"] = best_k
    out["smoothing_chosen"] = list(best_s)
    out["prolong_scale_chosen"] = best_w
    if rows["fcg_learned"]:
        out["speedup_learned_vs_plain_fcg"] = out["fcg"]["ms_mean"] / out["fcg_learned"]["ms_mean"]
        out["speedup_learned_vs_refine"] = out["refine"]["ms_mean"] / out["fcg_learned"]["ms_mean"]
    if rows["fcg_tuned_learned"]:
        tuned = out["fcg_fp16_c4_s11"]
        learned = out["fcg_tuned_learned"]
        out["learned_at_timed_settings"] = {
            "speedup": tuned["ms_mean"] / learned["ms_mean"], "ms_plain": tuned["ms_mean"],
            "ms_learned": learned["ms_mean"], "cycles_plain": tuned["cycles_mean"],
            "cycles_learned": learned["cycles_mean"],
            "cycles_saved_ms": (tuned["cycles_mean"] - learned["cycles_mean"]) * tuned["ms_mean"] /
            max(tuned["cycles_mean"], 1.0),
        }
    return out


def our_arm(args):
    import torch

    from continuum_liquid_b200 import scenes, solver
    from continuum_liquid_b200.backend import Backend
    from continuum_liquid_b200.replicas import ReplicaGroup, throughput

    group = ReplicaGroup("nccl")
    world, rank, local = group.world, group.rank, group.local_rank
    kernels = Backend(local)
    dev = kernels.device
    scene = scenes.block(args.size)
    obstacle = torch.zeros(scene.grid_shape, dtype=torch.uint8, device=dev)
    positions, velocities = scenes.seed_particles(scene)
    warm, warm_note = load_warm_start(kernels, scene, args.learned)
    opts = solver.StepOptions(flip_ratio=0.95, tol=TOL, gravity=scene.gravity, rho=scene.rho, nu=scene.nu,
                              method=args.method, warm_start=warm if args.learned == "on" else None)
    sim = solver.FlipSolver(kernels, scene.grid_shape, scene.dx, positions, velocities, obstacle=obstacle, dt=scene.dt,
                            options=opts, min_size=scene.min_size)
    n = sim.n
    parity = first_step_parity(sim, positions, velocities, scene) if rank == 0 else None

    barrier = group.barrier

    for _ in range(args.warmup):
        sim.step()
    torch.cuda.synchronize()

    # --- Poisson comparison on the next steps' systems; it also decides FP16 coarse storage ----
    poisson = {}
    use_fp16 = args.coarse_fp16 == "on"
    use_learned = args.learned == "on"
    coarse_k = COARSE_ITERATION_CHOICES[0] if args.coarse_iterations == "auto" else int(args.coarse_iterations)
    smoothing = SMOOTHING_CHOICES[0] if args.smoothing == "auto" else tuple(int(x) for x in args.smoothing.split(","))
    prolong = PROLONG_SCALE_CHOICES[0] if args.prolong_scale == "auto" else float(args.prolong_scale)
    coarse_smooth = None if args.coarse_smooth in ("auto", "none") else \
        tuple(int(x) for x in args.coarse_smooth.split(","))
    single_from = int(args.single_visit)
    if args.poisson_steps > 0:
        poisson.update(poisson_comparison(kernels, sim, args.poisson_steps, warm, scene.min_size))
        if args.coarse_fp16 == "auto":
            use_fp16 = poisson.get("coarse_fp16_chosen", poisson.get("coarse_fp16_holds", False))
        if args.coarse_iterations == "auto":
            coarse_k = poisson.get("coarse_iterations_chosen", coarse_k)
        if args.smoothing == "auto":
            smoothing = tuple(poisson.get("smoothing_chosen", smoothing))
        if args.prolong_scale == "auto":
            prolong = float(poisson.get("prolong_scale_chosen", prolong))
        if args.coarse_smooth == "auto" and poisson.get("coarse_smooth_chosen"):
            coarse_smooth = tuple(poisson["coarse_smooth_chosen"])
        if args.learned == "auto" and "fcg_tuned_learned" in poisson:
            # the rule: the learned guess in the timed steps only when it makes the solve faster,
            # network evaluation included
            use_learned = poisson["fcg_tuned_learned"]["ms_mean"] < poisson["fcg_fp16_c4_s11"]["ms_mean"]
    else:
        poisson["learned_vs_plain"] = "skipped (--poisson-steps 0)"
    sim.options.warm_start = warm if use_learned else None
    if warm is not None and not use_learned:
        warm_note += " (not used in the timed steps: no faster than without it in the comparison)"
    kernels.call("clb_mg_set_option", 4, single_from)  # read when the timed solver captures its graphs
    if use_fp16 or coarse_k != sim.options.coarse_iterations or single_from or \
            smoothing != (sim.options.pre_smooth, sim.options.post_smooth) or prolong != sim.options.prolong_scale or \
            coarse_smooth != sim.options.coarse_smooth:
        from continuum_liquid_b200.pressure_solve import PressureSolver

        sim.options.coarse_fp16 = use_fp16
        sim.options.coarse_iterations = coarse_k
        sim.options.pre_smooth, sim.options.post_smooth = smoothing
        sim.options.prolong_scale = prolong
        sim.options.coarse_smooth = coarse_smooth
        sim.pressure_solver = PressureSolver(kernels, sim.grid_shape, sim.dx, min_size=scene.min_size,
                                             method=args.method, coarse_fp16=use_fp16, coarse_iterations=coarse_k,
                                             pre_smooth=smoothing[0], post_smooth=smoothing[1], prolong_scale=prolong,
                                             coarse_smooth=coarse_smooth)
        for _ in range(2):  # tuning and graph capture of the new solver
            sim.step()
        torch.cuda.synchronize()

    # --- device-resident timed region -------------------------------------------------------
    snapshot = (sim.n, sim.particles[:n].clone(), sim.particle_velocity[:n].clone(), sim.pressure.clone())
    stats = []
    solve_ms = []
    launches0 = kernels.launch_count()
    replays0 = sim.pressure_solver.graph_replays
    loop0 = sim.pressure_solver.loop_refinements
    with ClockSampler(dev.index) as clocks:
        barrier()
        torch.cuda.synchronize()
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.nvtx.range_push("timed")
        start.record()
        for _ in range(args.steps):
            stats.append(sim.step())
        end.record()
        torch.cuda.nvtx.range_pop()
        torch.cuda.synchronize()
        barrier()
    clock_summary = clocks.summary()
    end_positions = sim.particles[:n].clone()
    value, elapsed_ms = throughput(group, args.steps, start.elapsed_time(end))
    direct_launches = kernels.launch_count() - launches0
    replays = sim.pressure_solver.graph_replays - replays0
    # refinements replayed from graphs (the host loop's or the device loop's), plus the device loop's
    # one check kernel per refinement
    gpu_launches = direct_launches + replays * sim.pressure_solver.graph_launches + \
        (sim.pressure_solver.loop_refinements - loop0)
    cycles = [s.cycles for s in stats]
    solve_ms = [s.device_ms() for s in stats]

    # --- Poisson time to 1e-6 in the timed steps ------------------------------------------------
    poisson = {"timed_steps": {"method": args.method, "learned": warm_note, "coarse_fp16": use_fp16,
                               "coarse_iterations": coarse_k, "smoothing": list(smoothing), "prolong_scale": prolong,
                               "coarse_smooth": list(coarse_smooth) if coarse_smooth else None,
                               "ms_mean": float(np.mean(solve_ms)),
                               "cycles_mean": float(np.mean(cycles)),
                               "final_rel_residual_max": float(max(s.rel_residual or 0.0 for s in stats)),
                               "initial_rel_residual_mean": float(np.mean([s.initial_rel_residual or 0.0
                                                                           for s in stats])),
                               "guess_used": sorted({s.warm_start for s in stats}),
                               "history_last_step": [float(x) for x in stats[-1].history]}, **poisson}

    # --- end to end through the stage API with host buffers ------------------------------------
    e2e = None
    if not args.no_e2e:
        host_pos = torch.empty((n, 3), dtype=torch.float32, pin_memory=True)
        host_vel = torch.empty((n, 3), dtype=torch.float32, pin_memory=True)
        host_pos.copy_(sim.particles[:n])
        host_vel.copy_(sim.particle_velocity[:n])
        torch.cuda.synchronize()
        barrier()
        s2, e2 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e2e_steps = max(1, args.steps)
        s2.record()
        for _ in range(e2e_steps):
            sim.step_host(host_pos, host_vel)
        e2.record()
        torch.cuda.synchronize()
        barrier()
        e2e_value, _ = throughput(group, e2e_steps, s2.elapsed_time(e2))
        e2e = {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": 24 * n,
               "d2h_bytes_per_step": 24 * n, "steps": e2e_steps,
               "path": "FlipSolver.step_host: the particle state copied from pinned host buffers before and back "
                       "after every step (the reference's per-step host round trip of solver.py:252-306), in 8 "
                       "pieces per direction on two copy streams: a piece's download starts once the particle "
                       "update of that piece is done and overlaps the next step's upload of earlier pieces"}

    # --- each timed step's pressure error against an FP64 reference solution (replayed steps) -------
    audit = pressure_error_audit(sim, snapshot, end_positions, args.steps, scene.min_size)
    del snapshot

    # --- roofline: the level-0 red-black sweep as the timed steps run it (on the fluid tiles), timed
    # alone on the stream ---------------------------------------------------------------------------
    ps = sim.pressure_solver
    h = ps.hierarchy
    iters = 20
    torch.cuda.synchronize()
    ps.correction.zero_()
    h.smooth(0, 2, ps.correction, ps.residual, zero_outside=True)
    s3, e3 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s3.record()
    h.smooth(0, iters, ps.correction, ps.residual, zero_outside=True)
    e3.record()
    torch.cuda.synchronize()
    per_launch_s = s3.elapsed_time(e3) / 1e3 / (2 * iters)
    vec = scene.grid_shape[2] % 4 == 0
    tiles0 = int(h.tile_counts[0].item())
    cells = tiles0 * 4 * (128 if vec else 32)  # the cells of the fluid tiles a launch streams
    # p read + write 8 B, b 4 B, packed operator 1 B per cell per red-black iteration; one colour per launch
    algorithmic = 13.0 * cells / 2.0
    achieved = algorithmic / per_launch_s / 1e9
    peak, peak_kind = measured_peak_hbm()
    kernel = "k_rbgs_colour_tiles<true,4>" if vec else "k_rbgs_colour_tiles<true,1>"
    traffic = NCU_TRAFFIC_BYTES.get(kernel)
    if traffic is not None and kernel in NCU_TILES_AT_CAPTURE:
        traffic = int(round(traffic * tiles0 / NCU_TILES_AT_CAPTURE[kernel]))
    roofline = {"kernel": f"{kernel} (level-0 red-black Gauss-Seidel on the {tiles0} fluid tiles of "
                          f"{int(h.kernels.lib.clb_mg_tile_capacity(*scene.grid_shape, 1))}, one colour per launch)",
                "bound": "hbm", "tile_cells": cells,
                "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "peak_source": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs)" if peak_kind == "measured" else "fallback",
                "traffic": traffic, "algorithmic_bytes_per_launch": algorithmic, "launch_us": per_launch_s * 1e6}

    rooflines = [dict(roofline, stage="level0_sweep", ms=per_launch_s * 1e3,
                      share_of_step=per_launch_s * 1e3 / (elapsed_ms / args.steps))]
    rooflines += kernel_rooflines(sim, peak, elapsed_ms / args.steps)

    # --- CPU baseline (rank 0, N = 1): the reference algorithm on the host cores ---------------
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        o = sim.options
        cpu_times, cpu_cycles = cpu_steps(cpu_sim(scene, positions, velocities, coarse_iterations=o.coarse_iterations,
                                                  pre_smooth=o.pre_smooth, post_smooth=o.post_smooth,
                                                  prolong_scale=o.prolong_scale, coarse_smooth=o.coarse_smooth), 1)
        cpu = {"value": 1.0 / cpu_times[0], "unit": UNIT, "cores": cpu_threads(), "kind": "port",
               "sample": f"the first step of the same scene ({n} particles) by the CPU restatement of the reference "
                         f"kernels, its pressure solved to {TOL:g} ({cpu_cycles[0]} cycles of the same iteration)"}

    if rank == 0:
        config = workload_config(args.size, n, args)
        fp16_levels = [list(s) for s in h.shapes[h.fp16_level:]] if h.fp16_level else None
        solver_info = {"pressure": solver_description(args.method, sim.options.pre_smooth, sim.options.post_smooth,
                                                      sim.options.coarse_iterations, fp16_levels, single_from,
                                                      sim.options.prolong_scale, sim.options.coarse_smooth),
                       "p2g": p2g_kernel(sim.options.tiled_p2g(), int(np.prod(sim.grid_shape))),
                       "multigrid_levels": [list(s) for s in h.shapes], "sweep_kinds": h.sweeps(),
                       "sweep_tuning_ms_per_iteration": h.tuning}
        line = {
            "metric": METRIC,
            "value": value,
            "unit": UNIT,
            "n_gpus": world,
            "steps": args.steps,
            "warmup": args.warmup,
            "ms_per_step": elapsed_ms / args.steps,
            "higher_is_better": True,
            "scaling": "weak",
            "vs_baseline": None,
            "dtype": "f32",
            "data": "synthetic",
            "config": config,
            "solver": solver_info,
            "particles_per_s": value * n,
            "parity": parity,
            "pressure_error": audit,
            "poisson": poisson,
            "e2e": e2e,
            "roofline": roofline,
            "rooflines": rooflines,
            "cpu_baseline": cpu,
            "clocks": clock_summary,
            "gpu_launches": int(gpu_launches),
        }
        short, details = printed_line(line)
        print(json.dumps({"details": details}), file=sys.stderr, flush=True)
        print(json.dumps(short), flush=True)
    group.close()


def main():
    args = parse_args()
    if args.impl == "reference":
        reference_arm(args)
    elif args.case in ("sweep0", "wcycle"):
        sweep_case(args)
    elif args.case == "batch":
        batch_case(args)
    elif args.case == "unet":
        unet_case(args)
    elif args.case == "collider":
        collider_case(args)
    elif args.case == "particles":
        particles_case(args)
    else:
        our_arm(args)


if __name__ == "__main__":
    main()
