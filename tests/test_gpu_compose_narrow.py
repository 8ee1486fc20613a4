"""lig_level_compose around the width up to which a CTA takes a whole row by several
groups of rows (128 values), at the edges of those groups."""
import pytest
import torch
import torch.nn.functional as F

from lig_b200.levels import compose

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1, 2, 5, 6, 11, 42, 43])
@pytest.mark.parametrize("h,ph,pw", [(1, 1, 1), (15, 15, None), (128, 61, 7), (145, 73, 22),
                                     (257, 300, 3), (1027, 9, 2)])
def test_narrow_rows(h, w, ph, pw):
    g = torch.Generator().manual_seed(h + w)
    render = (torch.rand(h, w, 3, generator=g) * 1.3 - 0.15).cuda()
    prev = torch.rand(ph, w if pw is None else pw, 3, generator=g).cuda()
    lo, hi = -0.25, 1.125
    est = torch.clamp(render, 0, 1) * (hi - lo) - 0.5 + lo
    up = F.interpolate(prev.permute(2, 0, 1)[None], size=(h, w), mode="bilinear")[0].permute(1, 2, 0)
    # a few float ulps at |values| <= 2.5 (contraction of the weights)
    assert (compose(prev, render, lo, hi, False) - (up + est)).abs().max().item() <= 4e-6
    assert torch.equal(compose(None, render, lo, hi, False), 0 + est)


@pytest.mark.parametrize("w", [2, 3, 11, 42])
def test_many_narrow_rows(w):
    """Rows enough for sixteen a group on every SM, the last CTA in part."""
    h, pw = 60001, (w + 1) // 2
    g = torch.Generator().manual_seed(w)
    render = (torch.rand(h, w, 3, generator=g) * 1.3 - 0.15).cuda()
    # (as many rows as the image: the source rows are whole numbers, no rounding in them)
    prev = torch.rand(h, pw, 3, generator=g).cuda()
    lo, hi = -0.25, 1.125
    est = torch.clamp(render, 0, 1) * (hi - lo) - 0.5 + lo
    up = F.interpolate(prev.permute(2, 0, 1)[None], size=(h, w), mode="bilinear")[0].permute(1, 2, 0)
    assert (compose(prev, render, lo, hi, False) - (up + est)).abs().max().item() <= 4e-6
