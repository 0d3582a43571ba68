"""Infinities and NaN in the weight gradient's input: an x value reaches the taps of the voxels next to it and nothing
else, also in the last column of a volume whose width is no multiple of a tile's 16 columns. Where the gradient is
finite its tolerance is that of FP32 sums (V eps times the sum of the products' magnitudes)."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 31, 33, 40])
@pytest.mark.parametrize("cin,cout,chunks", [(8, 16, 1), (40, 32, 9), (16, 64, 3), (64, 16, 40)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_wgrad_nonfinite_column(backend, W, cin, cout, chunks, value):
    B, D, H = 2, 3, 18
    g = torch.Generator().manual_seed(W * 100 + cin)
    x = torch.randn(B, D, H, W, cin, generator=g).to(torch.bfloat16)
    dy = torch.randn(B, D, H, W, cout, generator=g).to(torch.bfloat16)
    dy[dy == 0] = 0.5
    places = [(0, 1, 5, W - 1, 3), (1, 2, H - 1, W - 1, cin - 1), (0, 0, 0, W // 2, 6)]
    for b, z, y, c, i in places:
        x[b, z, y, c, i] = value
    got = torch.zeros(27 * cin, cout, device="cuda")
    backend.call("clb_conv3d_wgrad", x.cuda(), dy.cuda(), got, B, D, H, W, cin, cout, chunks)
    xp, dyd = F.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1)), dy.double()
    taps = [(a, b, c) for a in range(3) for b in range(3) for c in range(3)]
    def sums(xs, ds):
        return torch.cat([torch.einsum("bzyxi,bzyxo->io", xs[:, a:a + D, b:b + H, c:c + W], ds) for a, b, c in taps])
    # the pattern from the voxels that exist: which (tap, channel) sums hold a non-finite x
    bad = sums((~xp.isfinite()).double(), torch.ones_like(dyd)) > 0
    want = sums(torch.where(xp.isfinite(), xp, 0.0), dyd)
    size = sums(torch.where(xp.isfinite(), xp, 0.0).abs(), dyd.abs())
    got = got.cpu().double()
    assert bool((~got[bad].isfinite()).all())
    assert bool(got[~bad].isfinite().all())
    assert bool(((got - want).abs() <= B * D * H * W * 2.0**-23 * size)[~bad].all())
    assert backend.device_error() == 0
