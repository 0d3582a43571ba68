"""The marching weight gradient at the edges of its tiles (single slices, short last ranges, partial rows and
columns, channel counts in several chunks, an output that is not 16-byte aligned, added to what it holds) and the
bias gradient for channel counts with and without the shuffle path, against float64.

Tolerance: FP32 sums of V products, whose error is below V eps times the sum of their magnitudes."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def reference(x, dy, cin, cout):
    """[27 * cin, cout] sums over voxels, float64."""
    xp = F.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    D, H, W = x.shape[1:4]
    rows = [torch.einsum("bzyxi,bzyxo->io", xp[:, a:a + D, b:b + H, c:c + W], dy.double())
            for a in range(3) for b in range(3) for c in range(3)]
    return torch.cat(rows).reshape(27 * cin, cout)


@pytest.mark.parametrize("B,D,H,W,cin,cout,chunks,offset", [
    (1, 1, 1, 1, 8, 16, 1, 0), (1, 2, 17, 15, 16, 64, 3, 0), (2, 3, 16, 33, 24, 32, 1, 0), (1, 19, 5, 16, 40, 16, 2, 0),
    (1, 33, 18, 17, 96, 32, 40, 0), (40, 5, 20, 9, 16, 16, 9, 1), (3, 16, 31, 16, 64, 64, 11, 3), (1, 9, 64, 70, 8, 32, 1000, 0),
])
def test_wgrad_edges(backend, B, D, H, W, cin, cout, chunks, offset):
    g = torch.Generator().manual_seed(cin * 100 + D)
    x = torch.randn(B, D, H, W, cin, generator=g).to(torch.bfloat16)
    dy = torch.randn(B, D, H, W, cout, generator=g).to(torch.bfloat16)
    store = torch.full((27 * cin * cout + 8,), 0.5, device="cuda")
    dw = store[offset: offset + 27 * cin * cout].view(27 * cin, cout)
    backend.call("clb_conv3d_wgrad", x.cuda(), dy.cuda(), dw, B, D, H, W, cin, cout, chunks)
    want = 0.5 + reference(x, dy, cin, cout)
    bound = (B * D * H * W + 1) * 2.0**-23 * (0.5 + reference(x.abs(), dy.abs(), cin, cout))
    assert bool(((dw.cpu().double() - want).abs() <= bound).all())
    assert bool((store[:offset] == 0.5).all()) and bool((store[offset + 27 * cin * cout:] == 0.5).all())
    assert backend.device_error() == 0


@pytest.mark.parametrize("V,C", [(1, 16), (4097, 8), (100003, 24), (70001, 64), (333, 256), (5000, 104)])
def test_bias_grad(backend, V, C):
    g = torch.Generator().manual_seed(V)
    dy = torch.randn(V, C, generator=g).to(torch.bfloat16)
    db = torch.full((C,), -1.0, device="cuda")
    backend.call("clb_unet_bias_grad", dy.cuda(), db, V, C)
    want, size = dy.double().sum(0) - 1.0, dy.double().abs().sum(0) + 1.0
    assert bool(((db.cpu().double() - want).abs() <= (V + 1) * 2.0**-23 * size).all())
