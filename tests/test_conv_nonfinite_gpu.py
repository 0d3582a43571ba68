"""Infinite activations in the forward convolution and its data gradient: an infinite input makes the outputs that hold
it infinite, with the sign of its weight, and no other output. (Infinities lie too far apart to meet in one output.)"""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def kpad(k):
    return (k + 63) // 64 * 64


def infinite_in(shape, channels, g):
    x = torch.randn(*shape, channels, generator=g).to(torch.bfloat16)
    hot = torch.zeros(*shape, channels, dtype=torch.float64)
    B, D, H, W = shape
    n = 0
    for z in range(0, D, 3):
        for y in range(0, H, 3):
            for c in range(0, W, 3):
                hot[n % B, z, y, c, n % channels] = 1.0 if n % 2 else -1.0
                n += 1
    x[hot != 0] = (hot[hot != 0] * float("inf")).to(torch.bfloat16)
    return x, hot


def check(got, hot_out, finite_want, relu):
    want = torch.where(hot_out != 0, hot_out.sign() * float("inf"), finite_want)
    if relu:
        want = want.relu()
    inf = want.isinf()
    assert torch.equal(got[inf], want[inf])
    assert bool(((got - want).abs() <= 2.0**-7 * want.abs() + 1e-2)[~inf].all())


@pytest.mark.parametrize("shape", [(1, 4, 7, 9), (2, 3, 18, 17), (1, 9, 16, 16), (1, 2, 33, 8)])
@pytest.mark.parametrize("cin,cout", [(8, 16), (8, 32), (8, 64), (16, 16), (24, 32), (64, 64)])
def test_conv_infinite_activation(backend, shape, cin, cout):
    g = torch.Generator().manual_seed(cin + shape[2])
    w = (torch.randn(27 * cin, cout, generator=g) * (2.0 / (27 * cin)) ** 0.5).to(torch.bfloat16).float()
    w[w == 0] = 0.01
    kf, kd = kpad(27 * cin), kpad(27 * cout)
    wf = torch.empty(cout, kf, dtype=torch.bfloat16, device="cuda")
    wd = torch.empty(cin, kd, dtype=torch.bfloat16, device="cuda")
    backend.call("clb_conv3d_arrange_weights", w.cuda(), wf, wd, cin, cout, kf, kd)
    wt = w.to(torch.bfloat16).double().view(3, 3, 3, cin, cout).permute(4, 3, 0, 1, 2).contiguous()
    first = lambda t: t.permute(0, 4, 1, 2, 3)
    last = lambda t: t.permute(0, 2, 3, 4, 1)
    x, hot = infinite_in(shape, cin, g)
    cold = torch.where(x.isinf(), 0.0, x.double())
    for relu in (0, 1):
        y = torch.empty(*shape, cout, dtype=torch.bfloat16, device="cuda")
        backend.call("clb_conv3d_forward", x.cuda(), wf, None, y, *shape, cin, cout, kf, relu)
        check(y.cpu().double(), last(F.conv3d(first(hot), wt, padding=1)), last(F.conv3d(first(cold), wt, padding=1)), relu)
    if cin >= 16 and cin != 24:
        dy, hot = infinite_in(shape, cout, g)
        cold = torch.where(dy.isinf(), 0.0, dy.double())
        dx = torch.empty(*shape, cin, dtype=torch.bfloat16, device="cuda")
        backend.call("clb_conv3d_dgrad", dy.cuda(), wd, None, dx, *shape, cout, cin, kd)
        check(dx.cpu().double(), last(F.conv_transpose3d(first(hot), wt, padding=1)),
              last(F.conv_transpose3d(first(cold), wt, padding=1)), False)
    assert backend.device_error() == 0
