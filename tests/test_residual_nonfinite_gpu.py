"""The FP64 residual against the same sums in torch, term by term, with infinities and NaN in cells that a fluid cell's
operator does not weigh (the ghost layer, air above the surface) and in fluid cells: a product with weight 0 is formed
too, so the same residuals are NaN. Finite ones are equal bit for bit."""

import numpy as np
import pytest
import torch

from continuum_liquid_b200 import multigrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(12, 9, 14), (9, 20, 37), (10, 8, 260)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_residual_nonfinite(backend, shape, dtype):
    rng = np.random.default_rng(shape[2])
    ff = (rng.random(shape) > 0.3).astype(np.float32)
    ff[:, shape[1] // 2 + 1 :] = 0
    ff[[0, -1]] = 0
    ff[:, [0, -1]] = 0
    ff[:, :, [0, -1]] = 0
    dx = 1.0 / 64
    h = multigrid.MultigridHierarchy(backend, shape, dx)
    rhs = torch.zeros(shape, dtype=torch.float32, device="cuda")
    vel = [torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda() for _ in range(3)]
    h.rhs_operator(vel, torch.from_numpy(ff).cuda(), rhs, 1.0 / 240.0, 1000.0)
    p = torch.from_numpy(rng.standard_normal(shape)).to(dtype)
    for value in (float("inf"), float("-inf"), float("nan")):
        for _ in range(8):
            p[0, rng.integers(shape[1]), rng.integers(shape[2])] = value
            p[rng.integers(shape[0]), 0, rng.integers(shape[2])] = value
            p[rng.integers(shape[0]), rng.integers(shape[1]), -1] = value
            p[rng.integers(shape[0]), rng.integers(shape[1]), rng.integers(shape[2])] = value
    r = torch.full(shape, 5.0, dtype=torch.float32, device="cuda")
    norms = h.residual_norms(p.cuda(), rhs, r_out=r).cpu()
    op = h.op0.cpu().reshape(shape).to(torch.int64)
    inner = (slice(1, -1),) * 3
    at = lambda a, d, s: a[tuple(slice(1 + s, a.shape[q] - 1 + s) if q == d else slice(1, -1) for q in range(3))]
    pd = p.double()
    ws = 0.0
    for d in range(3):
        up = ((op[inner] >> (3 + d)) & 1).double() * at(pd, d, 1)
        down = ((at(op, d, -1) >> (3 + d)) & 1).double() * at(pd, d, -1)
        ws = up + down if d == 0 else ws + up + down
    delta = float(np.float32(dx))
    res = rhs.cpu()[inner].double() - (ws - (op[inner] & 7).double() * pd[inner]) * (1.0 / (delta * delta))
    fluid = (op[inner] & 64) != 0
    want = torch.zeros(shape)
    want[inner] = torch.where(fluid, res, 0.0).float()
    got = r.cpu()
    assert torch.equal(got.isnan(), want.isnan()) and bool(want.isnan().any()) and bool(want.isfinite().any())
    assert torch.equal(got[~want.isnan()], want[~want.isnan()])
    assert bool(norms[0].isnan())
    assert backend.device_error() == 0
