"""The culled voxelisation against the kernel that tests every triangle on every cell: bit for bit, on meshes
and on triangle soups with slivers, triangles larger than the domain, degenerate and non-finite ones."""

import numpy as np
import pytest
import torch

from continuum_liquid_b200 import scenes, voxelise_mesh

pytestmark = pytest.mark.gpu


def soup(rng, count, size, origin, extent):
    base = origin + rng.random((count, 1, 3)) * extent
    return (base + rng.normal(0, size, (count, 3, 3))).astype(np.float32)


@pytest.mark.parametrize("shape,scale,shift", [((9, 8, 17), 1.0, 0.0), ((31, 50, 23), 1.0, 100.0), ((64, 40, 33), 30.0, -7.0)])
def test_culled_matches_every_triangle(backend, shape, scale, shift):
    rng = np.random.default_rng(shape[0])
    delta = scale / max(shape)
    origin = np.array([-0.5 * shape[0] * delta + shift, -0.5 * shape[1] * delta, shift])
    extent = np.array(shape) * delta
    sets = [scenes.icosphere(3, 0.3 * scale, origin + extent * 0.45)]
    for size in (0.003, 0.05, 0.5, 4.0):
        sets.append(soup(rng, 700, size * scale, origin, extent))
    sliver = soup(rng, 600, 0.2 * scale, origin, extent)
    sliver[:, 2] = sliver[:, 0] + (sliver[:, 1] - sliver[:, 0]) * 0.5 + rng.normal(0, 1e-5 * scale, (600, 3)).astype(np.float32)
    d = np.asarray(backend.voxelise_direction, np.float32)
    grazing = soup(rng, 600, 0.2 * scale, origin, extent)  # nearly parallel to the rays: tiny determinants
    grazing[:, 1] = grazing[:, 0] + d * np.float32(0.4 * scale) + rng.normal(0, 1e-6 * scale, (600, 3)).astype(np.float32)
    odd = soup(rng, 40, 0.2 * scale, origin, extent)
    odd[0] = odd[0, :1]
    odd[1, 2] = np.nan
    odd[2, 0, 1] = np.inf
    odd[3, 1] = 3e38
    sets += [sliver, grazing, odd]
    for tris in sets:
        got = []
        for cull in (False, True):
            mask = torch.zeros(shape, dtype=torch.uint8, device="cuda")
            voxelise_mesh.voxelise_triangles(backend, None, tris, mask, shape, delta, origin, cull=cull)
            got.append(mask.cpu().numpy())
        assert np.array_equal(got[0], got[1])
