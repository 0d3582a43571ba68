"""The slice-marching convolution at the edges of its tiles: one and two column tiles, partial rows and columns,
single slices, several z blocks with a short last one, channel counts that need passes, half-used 16-channel
chunks and the 8-channel pairing. Against float64 on the same BF16 operands.

Tolerance: the result is rounded to BF16 once (2^-9 of its value) after FP32 accumulation, whose error is below
27 C eps times the sum of the magnitudes."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def kpad(k):
    return (k + 63) // 64 * 64


def check(got, want, magnitude, terms):
    bound = 2.0**-8 * want.abs() + terms * 2.0**-23 * magnitude + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("B,D,H,W,cin,cout", [
    (1, 1, 1, 1, 16, 16), (1, 1, 3, 9, 64, 64), (2, 2, 16, 8, 96, 32), (1, 17, 17, 15, 8, 16), (1, 35, 33, 18, 8, 32),
    (3, 33, 16, 17, 16, 16), (1, 9, 31, 24, 48, 16), (1, 11, 18, 33, 32, 64), (1, 8, 20, 7, 104, 16), (2, 6, 15, 16, 24, 64),
    (1, 5, 130, 40, 40, 32), (40, 3, 16, 16, 16, 32),
])
def test_conv_march_edges(backend, B, D, H, W, cin, cout):
    g = torch.Generator().manual_seed(D * 1000 + H * 10 + cin)
    x = torch.randn(B, D, H, W, cin, generator=g).to(torch.bfloat16)
    w = (torch.randn(27 * cin, cout, generator=g) * (2.0 / (27 * cin)) ** 0.5).to(torch.bfloat16).float()
    bias = torch.randn(cout, generator=g) * 0.1
    dy = torch.randn(B, D, H, W, cout, generator=g).to(torch.bfloat16)
    kf, kd = kpad(27 * cin), kpad(27 * cout)
    wf = torch.empty(cout, kf, dtype=torch.bfloat16, device="cuda")
    wd = torch.empty(cin, kd, dtype=torch.bfloat16, device="cuda")
    backend.call("clb_conv3d_arrange_weights", w.cuda(), wf, wd, cin, cout, kf, kd)
    wt = w.double().view(3, 3, 3, cin, cout).permute(4, 3, 0, 1, 2).contiguous()
    xr = x.double().permute(0, 4, 1, 2, 3)
    xd, dyd = x.cuda(), dy.cuda()
    for relu in (0, 1):
        y = torch.full((B, D, H, W, cout), float("nan"), dtype=torch.bfloat16, device="cuda")
        backend.call("clb_conv3d_forward", xd, wf, bias.cuda(), y, B, D, H, W, cin, cout, kf, relu)
        want = F.conv3d(xr, wt, bias.double(), padding=1)
        size = F.conv3d(xr.abs(), wt.abs(), bias.double().abs(), padding=1)
        check(y.cpu().permute(0, 4, 1, 2, 3), want.relu() if relu else want, size, 27 * cin)
    if cin in (16, 32, 48, 64, 96):
        dyr = dy.double().permute(0, 4, 1, 2, 3)
        want = F.conv_transpose3d(dyr, wt, padding=1)
        size = F.conv_transpose3d(dyr.abs(), wt.abs(), padding=1)
        for mask in (None, xd):
            dx = torch.full((B, D, H, W, cin), float("nan"), dtype=torch.bfloat16, device="cuda")
            backend.call("clb_conv3d_dgrad", dyd, wd, mask, dx, B, D, H, W, cout, cin, kd)
            ref = want if mask is None else want * (xr > 0)
            check(dx.cpu().permute(0, 4, 1, 2, 3), ref, size, 27 * cout)
    assert backend.device_error() == 0
