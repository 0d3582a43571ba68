"""Coarsest-level solves on slabs of a cluster (csrc/mg_coarse.cuh) against the single-block solve: W-cycles
agree bit for bit. Grids whose coarsest level takes one block with one and with two slots a thread, clusters
of several sizes up to 16, uneven slabs and one plane a slab; and a level whose planes are too large for a
slab, which is swept colour by colour."""

import numpy as np
import pytest
import torch

from continuum_liquid_b200 import multigrid

pytestmark = pytest.mark.gpu

F32 = np.float32

CASES = [
    ((14, 14, 14), (8, 8, 8), False),
    ((24, 25, 176), (8, 8, 46), False),
    ((32, 84, 65), (10, 23, 18), False),
    ((155, 27, 129), (41, 9, 34), False),
    ((27, 160, 160), (9, 42, 42), False),
    ((230, 230, 27), (59, 59, 9), False),
    ((27, 220, 220), (9, 57, 57), False),
    ((300, 300, 27), (77, 77, 9), False),
    ((24, 25, 176), (8, 8, 46), True),
    ((32, 84, 65), (10, 23, 18), True),
    ((27, 100, 99), (9, 27, 27), True),
]


@pytest.mark.parametrize("shape, coarsest, half", CASES)
def test_coarse_slabs_equal_single_block(backend, shape, coarsest, half):
    rng = np.random.default_rng(sum(shape))
    ff = (rng.random(shape) > 0.07).astype(F32)
    ff[shape[0] // 2 :, shape[1] // 2 :] = 0
    ff[[0, -1]] = 0
    ff[:, [0, -1]] = 0
    ff[:, :, [0, -1]] = 0
    vel = [torch.from_numpy(rng.standard_normal(shape).astype(F32)).cuda() for _ in range(3)]
    rhs = torch.zeros(shape, dtype=torch.float32, device="cuda")
    h = multigrid.MultigridHierarchy(backend, shape, 1.0 / 64, **({"fp16_max_size": 96} if half else {}))
    assert h.shapes[-1] == coarsest and h.is_fp16(h.levels - 1) == half
    h.rhs_operator(vel, torch.from_numpy(ff).cuda(), rhs, 1.0 / 240.0, 1000.0)
    h.build_coarse()
    h.residual_norms(torch.zeros_like(rhs), rhs)
    out = {}
    try:
        for slabs in (0, 1):
            backend.lib.clb_mg_set_option(0, 0)  # no one-launch visits: the coarsest level is solved by itself
            backend.lib.clb_mg_set_option(2, slabs)
            e = torch.zeros_like(rhs)
            for coarse_iterations in (64, 3):
                h.w_cycle(e, rhs, coarse_iterations=coarse_iterations)
            out[slabs] = (e, h.p[-1].clone())
    finally:
        backend.lib.clb_mg_set_option(2, 1)
        backend.lib.clb_mg_set_option(0, 1)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert out[1][1].abs().max() > 0
    assert backend.device_error() == 0
