"""Coarsest-level solves of few iterations, on both sides of the count from which the slab kernel is taken: W-cycles
agree bit for bit with those whose coarsest level never takes it."""

import numpy as np
import pytest
import torch

from continuum_liquid_b200 import multigrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(24, 24, 24), (30, 93, 34), (24, 25, 176), (32, 84, 65)])
@pytest.mark.parametrize("half", [False, True])
def test_few_iterations(backend, shape, half):
    rng = np.random.default_rng(sum(shape))
    ff = (rng.random(shape) > 0.1).astype(np.float32)
    for a in range(3):
        np.moveaxis(ff, a, 0)[[0, -1]] = 0
    vel = [torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda() for _ in range(3)]
    rhs = torch.zeros(shape, dtype=torch.float32, device="cuda")
    h = multigrid.MultigridHierarchy(backend, shape, 1.0 / 64, **({"fp16_max_size": 96} if half else {}))
    h.rhs_operator(vel, torch.from_numpy(ff).cuda(), rhs, 1.0 / 240.0, 1000.0)
    h.build_coarse()
    h.residual_norms(torch.zeros_like(rhs), rhs)
    for coarse in (0, 1, 2, 3, 4, 6):
        out = []
        try:
            for slabs in (0, 1):
                backend.lib.clb_mg_set_option(0, 0)  # no one-launch visits: the coarsest level is solved by itself
                backend.lib.clb_mg_set_option(2, slabs)
                e = torch.zeros_like(rhs)
                for _ in range(2):
                    h.w_cycle(e, rhs, pre_smooth=1, post_smooth=1, coarse_iterations=coarse)
                out.append((e, h.p[-1].clone()))
        finally:
            backend.lib.clb_mg_set_option(2, 1)
            backend.lib.clb_mg_set_option(0, 1)
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
        assert out[1][1].abs().max() > 0
    assert backend.device_error() == 0
