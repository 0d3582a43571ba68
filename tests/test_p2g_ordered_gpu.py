"""The reference-order P2G's tile walk against the oracle, bit for bit: the plane counts it chooses, extents that are
no multiple of a tile, rows with more particles than a staging buffer holds, particle arrays that do not start on a
16-byte boundary, clamped bins and empty tiles."""

import numpy as np
import pytest
import torch

from continuum_liquid_b200 import particles

pytestmark = pytest.mark.gpu


def run(backend, pos, vel, shape, dx, offset=0):
    n = len(pos)
    work, vwork, counts, outs, sums = particles.create_particle_sort_buffers(backend, shape, n)
    P, V = torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda()
    grid = [torch.full(shape, 7.0, dtype=torch.float32, device="cuda") for _ in range(4)]
    res = particles.particle_to_grid(backend, None, P, V, work, vwork, tuple(grid[:3]), counts, outs, sums, grid[3], n,
                                     shape, dx, 8)
    if offset:  # the sorted particles one float into larger buffers: no 16-byte boundary
        moved = []
        for t in res[:2]:
            m = torch.zeros(3 * n + offset, dtype=torch.float32, device="cuda")
            m[offset:] = t.reshape(-1)
            moved.append(m[offset:].view(n, 3))
        grid = [torch.full(shape, 7.0, dtype=torch.float32, device="cuda") for _ in range(4)]
        particles.particle_to_grid_gather(backend, None, *moved, outs[0], counts, tuple(grid[:3]), grid[3], shape, dx, 8)
    return [g.cpu().numpy() for g in grid]


@pytest.mark.parametrize("shape,count", [((33, 64, 63), 60000), ((130, 29, 35), 40000), ((70, 80, 95), 120000),
                                         ((41, 200, 150), 150000)])
@pytest.mark.parametrize("offset", [0, 1])
def test_tile_walk_matches_oracle(backend, oracle, shape, count, offset):
    rng = np.random.default_rng(shape[0])
    dx = np.float32(1.0 / 64)
    extent = np.array(shape) * dx
    block = (0.1 + 0.6 * rng.random((count, 3))) * extent
    dense = (np.array([9.5, 11.5, 12.0]) + rng.random((900, 3)) * [1.0, 1.0, 25.0]) * dx  # rows of hundreds
    pile = (np.array([20.6, 20.6, 20.6]) + rng.random((700, 3)) * 0.3) * dx               # one bin of hundreds
    outside = np.array([[-0.2, 0.5, 0.5], [0.5, 50.0, 0.3], [0.3, 0.2, -3.0]])
    corners = rng.integers(0, 2, (200, 3)) * (extent - 2.2 * dx) + 1.1 * dx
    pos = np.concatenate([block, dense, pile, outside, corners]).astype(np.float32)
    vel = rng.standard_normal(pos.shape).astype(np.float32)
    _, _, u, v, w, ff, _, _ = oracle.particle_to_grid(pos, vel, dx, shape)
    for got, want in zip(run(backend, pos, vel, shape, float(dx), offset), (u, v, w, ff)):
        assert np.array_equal(got, want)
    assert backend.device_error() == 0
