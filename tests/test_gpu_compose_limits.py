"""lig_level_compose on an image of more rows than 65535 blocks of sixteen hold.
Without a resize the sums are those of the torch expression, bit for bit; with
one, prev is so smooth that the rounding of a large source row (2^-5 of a row)
moves the result by less than a float ulp of the values."""
import pytest
import torch
import torch.nn.functional as F

from lig_b200.levels import compose

pytestmark = pytest.mark.gpu

LO, HI = -0.25, 1.125


def _est(render):
    return torch.clamp(render, 0, 1) * (HI - LO) - 0.5 + LO


@pytest.mark.parametrize("resize", [False, True])
@pytest.mark.parametrize("H", [1048560, 1048561, 2100003])
def test_tall_image(H, resize):
    render = torch.rand(H, 1, 3, generator=torch.Generator().manual_seed(1)).cuda()
    assert torch.equal(compose(None, render, LO, HI, False), 0 + _est(render))
    ph = (H + 1) // 2 if resize else H
    prev = (torch.arange(ph, device="cuda").view(-1, 1, 1) / ph
            + torch.arange(3, device="cuda")).contiguous()
    up = prev
    if resize:
        up = F.interpolate(prev.permute(2, 0, 1)[None], size=(H, 1), mode="bilinear")
        up = up[0].permute(1, 2, 0)
    out = compose(prev, render, LO, HI, True)
    assert (out - torch.clamp(up + _est(render), 0, 1)).abs().max().item() <= 4e-6
