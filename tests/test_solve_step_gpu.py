"""The refinement and flexible-CG steps in one launch (small grids) and in two (large ones), on both sides of the sizes
that choose, rows that are and are not a multiple of 4 cells: pressure, direction and residual equal the same operations
in torch bit for bit; the sums of squares agree to FP64 rounding."""

import numpy as np
import pytest
import torch

from continuum_liquid_b200 import multigrid

pytestmark = pytest.mark.gpu


def residual(op, p, b, delta):
    inner = (slice(1, -1),) * 3
    at = lambda a, d, s: a[tuple(slice(1 + s, a.shape[q] - 1 + s) if q == d else slice(1, -1) for q in range(3))]
    ws = None
    for d in range(3):
        up = ((op[inner] >> (3 + d)) & 1).double() * at(p, d, 1)
        down = ((at(op, d, -1) >> (3 + d)) & 1).double() * at(p, d, -1)
        ws = up + down if ws is None else ws + up + down
    res = b[inner].double() - (ws - (op[inner] & 7).double() * p[inner]) * (1.0 / (delta * delta))
    out = torch.zeros_like(p)
    out[inner] = torch.where((op[inner] & 64) != 0, res, 0.0)
    return out


FCG, IR = "fcg", "ir"


@pytest.mark.parametrize("method,shape,launches", [
    (FCG, (3, 3, 3), 2), (FCG, (27, 37, 36), 2), (FCG, (60, 50, 100), 2), (FCG, (60, 50, 101), 3), (FCG, (41, 90, 84), 3),
    (FCG, (20, 60, 270), 3), (IR, (27, 37, 35), 2), (IR, (40, 200, 300), 2), (IR, (150, 200, 150), 2), (IR, (150, 200, 151), 3),
    (IR, (165, 166, 168), 3),
])
@pytest.mark.parametrize("skip", [0, 1])
def test_step_matches(backend, method, shape, launches, skip):
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(shape[2])
    ff = (torch.rand(shape, generator=g, device=dev) > 0.2).float()
    ff[:, shape[1] // 2 + 1 :] = 0
    for a in range(3):
        ff.select(a, 0).zero_()
        ff.select(a, -1).zero_()
    dx = 1.0 / 64
    delta = float(np.float32(dx))
    h = multigrid.MultigridHierarchy(backend, shape, dx)
    rhs = torch.zeros(shape, device=dev)
    vel = [torch.randn(shape, generator=g, device=dev) for _ in range(3)]
    h.rhs_operator(vel, ff, rhs, 1.0 / 240.0, 1000.0)
    op = h.op0.view(shape).long()
    fluid = (op & 64) != 0
    e = torch.where(fluid, torch.randn(shape, generator=g, device=dev), 0.0)
    d_in = torch.where(fluid, torch.randn(shape, generator=g, device=dev), 0.0)
    p_in = torch.where(fluid, torch.randn(shape, generator=g, device=dev, dtype=torch.float64), 0.0)
    state = torch.tensor([0.37, -1.21, 0.0, 0.0], dtype=torch.float64, device=dev)
    p_out, d_out, r = torch.zeros_like(p_in), torch.zeros_like(d_in), torch.zeros_like(rhs)
    norms = torch.zeros(2, dtype=torch.float64, device=dev)
    try:
        backend.lib.clb_mg_set_option(3, skip)
        before = backend.launch_count()
        if method == FCG:
            backend.call("clb_mg_fcg_step", p_in, e, d_in, p_out, d_out, state, rhs, h.op0, delta, *shape, r, h.partials,
                         norms)
            d = (e.double() + state[1] * d_in.double()).float()
            p = p_in + state[0] * d.double()
        else:
            backend.call("clb_mg_ir_step", p_in, e, p_out, rhs, h.op0, delta, *shape, r, h.partials, norms)
            d = d_out
            p = p_in + e.double()
        count = backend.launch_count() - before
    finally:
        backend.lib.clb_mg_set_option(3, 1)
    want = residual(op, p, rhs, delta)
    assert count == launches
    assert torch.equal(p_out, p) and torch.equal(d_out, d) and torch.equal(r, want.float())
    sums = torch.stack([(want * want).sum(), (rhs.double() ** 2)[fluid].sum()])
    assert bool(((norms - sums).abs() <= 1e-12 * sums).all())
    assert backend.device_error() == 0
