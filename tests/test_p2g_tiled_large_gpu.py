"""The tiled P2G on grids large enough to take it (3.5M cells and more), sparsely filled so that the oracle stays cheap:
extents that are no multiple of a tile, rows and bins of hundreds of particles, clamped and corner bins, particle arrays
that do not start on a 16-byte boundary; one cell count below the limit, where the reference-order walk runs; and a batch
of scenes on both sides of the limit.

Tolerance: a face's value is a quotient of two sums of n terms; their order and rounding may change it by 2 (n + 4) eps
times the largest speed among the terms, on either side (n: the particles in the bins around the face)."""

import numpy as np
import pytest
import torch

from continuum_liquid_b200 import batch, particles, scenes, solver

pytestmark = pytest.mark.gpu


def inputs(shape, dx, rng):
    extent = np.array(shape) * dx
    block = (np.array([0.4, 0.1, 0.2]) + 0.12 * rng.random((60000, 3))) * extent
    dense = (np.array([9.5, 11.5, 12.0]) + rng.random((900, 3)) * [1.0, 1.0, 25.0]) * dx  # rows of hundreds
    pile = (np.array([20.6, 20.6, 20.6]) + rng.random((700, 3)) * 0.3) * dx               # one bin of hundreds
    piles = (np.array([30.6, 40.6, 50.6]) + rng.random((2000, 3)) * [0.8, 0.8, 6.0]) * dx  # some in a row
    outside = np.array([[-0.2, 0.5, 0.5], [0.5, 50.0, 0.3], [0.3, 0.2, -3.0]])
    corners = rng.integers(0, 2, (200, 3)) * (extent - 2.2 * dx) + 1.1 * dx
    pos = np.concatenate([block, dense, pile, piles, outside, corners]).astype(np.float32)
    return pos, rng.standard_normal(pos.shape).astype(np.float32)


def around(shape, pos, dx):
    """Particles in the 3 x 3 x 3 bins around each cell."""
    n = np.zeros(shape)
    b = np.clip(np.floor(pos / dx - 0.5).astype(int), 0, np.array(shape) - 2)
    np.add.at(n, tuple(b.T), 1)
    for a in range(3):
        n = sum(np.roll(n, k, a) for k in (-1, 0, 1))
    return n


@pytest.mark.parametrize("shape,tiled_kernel", [((131, 173, 157), True), ((350, 101, 100), True), ((100, 101, 350), True),
                                                ((350, 100, 99), False)])
@pytest.mark.parametrize("offset", [0, 1])
def test_tiled_matches_oracle(backend, oracle, shape, tiled_kernel, offset):
    rng = np.random.default_rng(shape[0])
    dx = np.float32(1.0 / 64)
    pos, vel = inputs(shape, dx, rng)
    n = len(pos)
    work, vwork, counts, outs, sums = particles.create_particle_sort_buffers(backend, shape, n)
    P, V = torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda()
    grid = [torch.full(shape, 7.0, dtype=torch.float32, device="cuda") for _ in range(4)]
    res = particles.particle_to_grid(backend, None, P, V, work, vwork, tuple(grid[:3]), counts, outs, sums, grid[3], n,
                                     shape, float(dx), 8)
    ordered = [g.cpu().numpy() for g in grid]
    sorted_ = []
    for t in res[:2]:  # the sorted records `offset` floats into larger buffers
        m = torch.zeros(3 * n + offset, dtype=torch.float32, device="cuda")
        m[offset:] = t.reshape(-1)
        sorted_.append(m[offset:].view(n, 3))
    runs = []
    for _ in range(2):
        grid = [torch.full(shape, 7.0, dtype=torch.float32, device="cuda") for _ in range(4)]
        particles.particle_to_grid_gather(backend, None, *sorted_, outs[0], counts, tuple(grid[:3]), grid[3], shape,
                                          float(dx), 8, tiled=True)
        runs.append([g.cpu().numpy() for g in grid])
    _, _, u, v, w, ff, _, _ = oracle.particle_to_grid(pos, vel, dx, shape)
    bound = 2 * (around(shape, pos, dx) + 4) * 2.0**-23 * np.abs(vel).max()
    assert np.array_equal(runs[0][3], ff)
    for got, again, want, plain in zip(runs[0], runs[1], (u, v, w), ordered):
        assert np.array_equal(got, again)
        assert np.array_equal(plain, want)
        assert bool((np.abs(got.astype(np.float64) - want) <= bound).all())
        assert np.array_equal(got == 0, want == 0)
        assert np.array_equal(got, want) != tiled_kernel  # the tiled kernel's order rounds some faces differently
    assert backend.device_error() == 0


@pytest.mark.parametrize("tiled", [True, False])
def test_batch_with_a_large_scene(backend, tiled):
    several = [scenes.dam_break(24, seed=1), scenes.dam_break(30, seed=2), scenes.dam_break(20, seed=3)]
    several[1].grid_shape = (162, 150, 147)
    tol = 1e-6 if tiled else None
    b = batch.BatchedFlip(backend, several, flip_ratio=0.95, tol=tol, use_graph=False)
    assert b.batch.p2g_tiled == int(tiled)
    b.pre_solve()
    host = lambda t: t.detach().cpu().numpy()  # noqa: E731
    for s, scene in enumerate(several):
        pos, vel = scenes.seed_particles(scene)
        opts = solver.StepOptions(flip_ratio=0.95, tol=tol, gravity=scene.gravity, use_graph=False)
        sim = solver.FlipSolver(backend, scene.grid_shape, scene.dx, pos, vel, dt=scene.dt, options=opts)
        sim.pre_solve()
        for got, want, name in ((b.u, sim.u, "u"), (b.v, sim.v, "v"), (b.w, sim.w, "w"),
                                (b.fluid_fraction, sim.fluid_fraction, "fluid fraction")):
            assert np.array_equal(host(b.scene_view(got, s)), host(want)), (s, name)
    assert backend.device_error() == 0
