"""Residual target and compose at the edges of their vector and row split:
sizes that are no multiple of four values, arrays that start off a 16-byte
boundary (scalar path), rows past a CTA's sixteen, same-size and absent
previous levels."""
import pytest
import torch
import torch.nn.functional as F

from lig_b200.levels import compose, residual_target

pytestmark = pytest.mark.gpu


def _image(h, w, offset, seed):
    """[h, w, 3] contiguous, its first value `offset` floats into an allocation."""
    g = torch.Generator().manual_seed(seed)
    buf = torch.empty(h * w * 3 + 8, device="cuda")
    img = buf[offset:offset + h * w * 3].view(h, w, 3)
    img.copy_(torch.rand(h, w, 3, generator=g) * 1.3 - 0.15)
    return img


@pytest.mark.parametrize("h,w", [(1, 1), (1, 2), (33, 517), (64, 64), (301, 1203)])
@pytest.mark.parametrize("offsets", [(0, 0), (1, 0), (3, 3)])
def test_residual_bit_identical(h, w, offsets):
    gt, up = _image(h, w, offsets[0], 1), _image(h, w, offsets[1], 2)
    t, lo, hi = residual_target(gt, up)
    r = gt - up + 0.5
    assert torch.equal(lo, r.min()) and torch.equal(hi, r.max())
    assert torch.equal(t, (r - lo) / (hi - lo))


@pytest.mark.parametrize("prev_hw,hw", [((8, 9), (16, 86)), ((9, 43), (17, 85)), ((20, 20), (3, 171)),
                                        ((1, 1), (35, 4)), ((33, 29), (33, 29)), (None, (18, 90))])
@pytest.mark.parametrize("offset", [0, 1])
def test_compose_row_split(prev_hw, hw, offset):
    render = _image(*hw, offset, 3)
    lo, hi = -0.25, 1.125
    est = torch.clamp(render, 0, 1) * (hi - lo) - 0.5 + lo
    if prev_hw is None:
        prev, up = None, 0.0
    else:
        prev = _image(*prev_hw, offset, 4)
        up = F.interpolate(prev.permute(2, 0, 1)[None], size=hw, mode="bilinear")[0].permute(1, 2, 0)
    for last in (False, True):
        out = compose(prev, render, lo, hi, last)
        exp = torch.clamp(up + est, 0, 1) if last else up + est
        # a few float ulps at |values| <= 2.5 (contraction of the weights)
        assert (out - exp).abs().max().item() <= 4e-6
