"""The upscale over a reversed ROI (x2 < x1 and / or y2 < y1: a mirrored crop):
forward and backward against the C oracle, which gathers and scatters in the
order of the outputs.  Tolerances as in the upscale kernels' other tests."""
import numpy as np
import pytest
import torch

from lig_b200 import ops
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [  # src h, w -> dst h, w, roi
    (13, 11, 30, 27, (9.0, 2.0, 2.0, 11.0)),
    (13, 11, 30, 27, (2.0, 11.0, 9.0, 2.0)),
    (40, 50, 80, 120, (45.0, 33.0, 2.0, 3.0)),
    (40, 50, 31, 23, (50.0, 0.0, 0.0, 40.0)),       # down-scaling
    (12, 20, 90, 300, (15.0, 10.0, 5.0, 2.0)),      # more than eight columns a texel
    (20, 90, 45, 200, (100.0, 25.0, 0.0, 0.0)),  # past the border, two CTAs a row
]


@pytest.mark.parametrize("ch", [3, 1])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}-{c[2]}x{c[3]}")
def test_reversed_roi(case, ch):
    h, w, dh, dw, roi = case
    g = torch.Generator().manual_seed(h * 31 + w)
    planes = [torch.rand(h, w, ch, generator=g, dtype=torch.float64) for _ in range(4)]
    cot = torch.rand(dh, dw, ch, generator=g, dtype=torch.float64)
    three = [np.repeat(p.numpy(), 3 // ch, axis=2) for p in planes + [cot]]
    exp = O.upscale_fwd(*three[:4], dh, dw, roi=roi, dtype=np.float64)[..., :ch]
    eg = [x[..., :ch] for x in O.upscale_bwd(three[4], h, w, roi=roi, dtype=np.float64)]
    for dt, tol in ((torch.float64, 1e-11), (torch.float32, 2e-4)):
        got = ops.upscale_fwd(*[p.to("cuda", dt) for p in planes], dh, dw, roi, 0)
        assert np.abs(got.cpu().numpy() - exp).max() <= tol
        gg = ops.upscale_bwd(cot.to("cuda", dt), h, w, roi, 0)
        for a, b in zip(gg, eg):
            assert np.abs(a.cpu().numpy() - b).max() <= tol * max(1.0, np.abs(b).max())
