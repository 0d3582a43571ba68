"""The weight gradient's promise on precision: no tensor-core sum is longer than chunks_per_block chunks of 64 voxels.

x is 1 everywhere, so the centre tap's gradient is the sum of dy over all voxels. dy is 2^24 at one voxel and 2^-5
at the others: a row of 16 of those (0.5) is lost where it is added to the sum that holds 2^24 (spacing 2), and every
other sum of whole rows of 64 voxels is an even number, exact in FP32 in any order. So what may be missing is at most the sum
that holds the large value: 64 chunks_per_block terms of 2^-5."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [1, 2, 3, 4, 5, 7, 8, 12])
@pytest.mark.parametrize("B,D,cin,cout", [(1, 4, 16, 16), (64, 8, 16, 16), (64, 8, 40, 32), (2, 3, 96, 64)])
def test_sums_are_no_longer_than_asked(backend, B, D, cin, cout, chunks):
    H = W = 16
    small = 2.0**-5
    x = torch.ones(B, D, H, W, cin, dtype=torch.bfloat16, device="cuda")
    dy = torch.full((B, D, H, W, cout), small, dtype=torch.bfloat16, device="cuda")
    dy[0, 1, 0, 0] = 2.0**24
    dw = torch.zeros(27 * cin, cout, device="cuda")
    backend.call("clb_conv3d_wgrad", x, dy, dw, B, D, H, W, cin, cout, chunks)
    rest = (dw.view(27, cin, cout)[13].double() - 2.0**24).cpu()
    exact = (B * D * H * W - 1) * small
    assert bool((rest >= exact - 64 * chunks * small).all()) and bool((rest <= exact + 2.0).all())
    assert backend.device_error() == 0
