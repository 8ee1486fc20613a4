"""Residual target of large arrays that start off a 16-byte boundary (images of
odd size inside a batch, rows of an odd-sized image): values one at a time on
more CTAs than the vector passes."""
import pytest
import torch

from lig_b200.levels import residual_target

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(1414, 1414), (1415, 1415), (2049, 2047)])  # 6M values between
@pytest.mark.parametrize("off_gt,off_up", [(1, 0), (3, 2)])
def test_residual_bit_identical(h, w, off_gt, off_up):
    g = torch.Generator(device="cuda").manual_seed(1)
    n = 3 * h * w

    def image(off):
        return torch.rand(n + 4, generator=g, device="cuda")[off:off + n].view(h, w, 3)

    gt, up = image(off_gt), image(off_up)
    t, lo, hi = residual_target(gt, up)
    r = gt - up + 0.5
    assert torch.equal(lo, r.min()) and torch.equal(hi, r.max())
    assert torch.equal(t, (r - lo) / (hi - lo))
