"""The upscale backward with more than eight output columns a texel (a warp per
texel column, but for a few more columns of a large source) against the C oracle: around ten, twenty and forty columns (three
channels) and 32 and 64 (one), more than a warp takes in one walk, source widths
around the warps of a CTA, one and several texel rows a warp, both coordinate
maps and ROIs.  Tolerances as in the upscale kernels' other tests."""
import numpy as np
import pytest
import torch

from lig_b200 import ops
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [  # src h, w -> dst h, w, roi, mode
    (3, 7, 15, 32, None, 0),                          # nine or ten columns
    (5, 8, 9, 40, None, 0),                           # ten
    (2, 9, 20, 90, None, 0),                          # twenty
    (9, 17, 40, 175, None, 0),                        # twenty or twenty-one
    (1, 5, 3, 100, None, 0),                          # forty
    (4, 3, 7, 65, None, 0),                           # 43
    (2, 2, 11, 200, None, 0),                         # 200: five walks
    (6, 4, 30, 61, None, 1),
    (1, 1, 5, 40, None, 1),                           # every corner clamped
    (30, 40, 64, 90, (10.0, 4.0, 24.0, 20.0), 0),     # a crop: texels without outputs
    (30, 40, 64, 90, (24.0, 4.0, 10.0, 20.0), 0),     # reversed
    (200, 200, 300, 1000, None, 0),                   # eight texel rows a warp
    (460, 460, 500, 2300, None, 0),                   # ten, but a thread a value
]


@pytest.mark.parametrize("ch", [3, 1])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}-{c[2]}x{c[3]}-m{c[5]}")
def test_strong_upscale_backward(case, ch):
    h, w, dh, dw, roi, mode = case
    g = torch.Generator().manual_seed(h * 31 + w)
    cot = torch.rand(dh, dw, ch, generator=g, dtype=torch.float64)
    three = np.repeat(cot.numpy(), 3 // ch, axis=2)  # the oracle takes three channels
    exp = [x[..., :ch] for x in O.upscale_bwd(three, h, w, roi=roi, mode=mode, dtype=np.float64)]
    for dt, tol in ((torch.float64, 1e-11), (torch.float32, 2e-4)):
        got = ops.upscale_bwd(cot.to("cuda", dt), h, w, roi, mode)
        for a, b in zip(got, exp):
            assert np.abs(a.cpu().numpy() - b).max() <= tol * max(1.0, np.abs(b).max())


def test_non_finite_cotangents_stay_in_their_cell():
    h, w, dh, dw = 4, 5, 30, 50
    for j, i in ((0, 0), (2, 7), (29, 49), (15, 24)):
        cot = torch.zeros(dh, dw, 3)
        cot[j, i, 1] = float("nan")
        exp = O.upscale_bwd(cot.numpy(), h, w, mode=0, dtype=np.float32)
        for a, b in zip(ops.upscale_bwd(cot.cuda(), h, w, None, 0), exp):
            assert np.array_equal(np.isnan(a.cpu().numpy()), np.isnan(b))
