"""The particle update by tiles on small and odd grids, below the particle count from which it is taken by itself: records
that start 4 bytes off a 16-byte boundary take it at any count. Bit for bit the per-particle kernel's values, with and
without an obstacle, moving or not, with empty tiles and partly filled ones, rows of hundreds and clamped particles."""

import numpy as np
import pytest
import torch

from continuum_liquid_b200 import particles as pm
from continuum_liquid_b200.colliders import RigidMotion

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 9, 31), (37, 45, 71), (20, 64, 33), (41, 18, 95)])
@pytest.mark.parametrize("obstacle", ["none", "still", "moving"])
@pytest.mark.parametrize("previous", [False, True])
def test_tiles_match_per_particle(backend, shape, obstacle, previous):
    rng = np.random.default_rng(shape[2])
    dev = backend.device
    dx = np.float32(1.0 / 64)
    extent = np.array(shape) * dx
    pos = np.concatenate([
        (np.array([0.1, 0.2, 0.05]) + np.array([0.35, 0.5, 0.6]) * rng.random((4000, 3))) * extent,
        (np.array([5.6, 5.6, 5.6]) + 0.3 * rng.random((700, 3))) * dx,
        rng.integers(0, 2, (100, 3)) * (extent - 2.2 * dx) + 1.1 * dx,
        np.array([[-0.2, 0.05, 0.05], [0.05, 50.0, 0.03], [0.03, 0.02, -3.0]]),
    ]).astype(np.float32)
    vel = (rng.standard_normal(pos.shape) * 2.0).astype(np.float32)
    n = len(pos)
    P, V = torch.from_numpy(pos).to(dev), torch.from_numpy(vel).to(dev)
    work, vwork, counts, outputs, sums = pm.create_particle_sort_buffers(backend, shape, n)
    grid = [torch.zeros(shape, dtype=torch.float32, device=dev) for _ in range(4)]
    pm.particle_to_grid(backend, None, P, V, work, vwork, tuple(grid[:3]), counts, outputs, sums, grid[3], n, shape,
                        float(dx), 8)
    cur, old = ([torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).to(dev) for _ in range(3)] for _ in range(2))
    solid = None if obstacle == "none" else torch.from_numpy((rng.random(shape) < 0.2).astype(np.uint8)).to(dev)
    motion = None
    if obstacle == "moving":
        motion = RigidMotion(velocity=(0.3, -0.2, 0.1), angular_velocity=(0.0, 1.5, 0.5),
                             pivot=(0.2, 0.1, 0.3)).parameters(0.01, (0.0, 0.0, 0.0))
    results = []
    for offset in (0, 1):
        records = []
        for t in (work, vwork):
            flat = torch.empty(3 * n + 4, dtype=torch.float32, device=dev)
            view = flat[offset:offset + 3 * n].view(n, 3)
            view.copy_(t[:n])
            records.append(view)
        prev = torch.zeros_like(work[:n]) if previous else None
        pm.particle_update(backend, None, *records, tuple(cur), tuple(old), solid, n, shape, float(dx), 1.0 / 240.0,
                           flip_ratio=0.95, previous_particles=prev, motion=motion,
                           bins=(outputs[0], counts) if offset else None)
        results.append(records + ([prev] if previous else []))
    for a, b in zip(*results):
        assert torch.equal(a.contiguous().view(torch.int32), b.contiguous().view(torch.int32))
    assert not torch.equal(results[1][0], work[:n])
    assert backend.device_error() == 0
