"""Upscale kernels at the edges of their split (256 values of a row per CTA,
8..64 rows per CTA, a 1024-column weight table) against the C oracle: up- and
down-scaling, odd sizes, ROI, both coordinate maps, one and three channels.

The double instantiation runs the same code: both sides form the same sums of
at most a few hundred products of O(1) values, so they agree to 1e-11.  In
float the coordinate s has an error of a few ulp (s <= 64 here: below 3e-5)
and the weights' slopes are below 2, with planes in [0, 1]."""
import numpy as np
import pytest
import torch

from lig_b200 import ops
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [  # src h, w -> dst h, w, roi, mode
    (3, 5, 9, 20, None, 0),
    (16, 43, 64, 172, None, 0),            # 516 values a row: a ragged third CTA
    (17, 64, 65, 256, None, 1),            # 768 values a row: full CTAs only
    (40, 33, 8, 7, None, 0),               # down-scaling: rows and columns skipped
    (9, 64, 130, 2000, None, 0),           # more than 1024 columns behind a CTA's texels
    (64, 50, 63, 101, (3.25, 7.5, 41.0, 60.0), 0),
    (1, 1, 4, 6, None, 0),                 # every corner clamped
    (5, 2, 1, 1, None, 1),
]


@pytest.mark.parametrize("ch", [3, 1])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}-{c[2]}x{c[3]}-m{c[5]}")
def test_upscale_split_edges(case, ch):
    h, w, dh, dw, roi, mode = case
    g = torch.Generator().manual_seed(h * 31 + w)
    planes = [torch.rand(h, w, ch, generator=g, dtype=torch.float64) for _ in range(4)]
    cot = torch.rand(dh, dw, ch, generator=g, dtype=torch.float64)
    # the oracle takes three channels
    three = [np.repeat(p.numpy(), 3 // ch, axis=2) for p in planes + [cot]]
    exp = O.upscale_fwd(*three[:4], dh, dw, roi=roi, mode=mode, dtype=np.float64)[..., :ch]
    eg = [x[..., :ch] for x in O.upscale_bwd(three[4], h, w, roi=roi, mode=mode,
                                             dtype=np.float64)]
    for dt, tol in ((torch.float64, 1e-11), (torch.float32, 2e-4)):
        got = ops.upscale_fwd(*[p.to("cuda", dt) for p in planes], dh, dw, roi, mode)
        assert np.abs(got.cpu().numpy() - exp).max() <= tol
        gg = ops.upscale_bwd(cot.to("cuda", dt), h, w, roi, mode)
        for a, b in zip(gg, eg):
            assert np.abs(a.cpu().numpy() - b).max() <= tol * max(1.0, np.abs(b).max())


def test_upscale_backward_keeps_non_finite_cotangents_to_their_texels():
    """A NaN cotangent reaches exactly the (at most four) texels of its cell."""
    h, w, dh, dw = 6, 7, 12, 14
    for j, i in ((0, 0), (0, 5), (11, 13), (6, 7)):
        cot = torch.zeros(dh, dw, 3)
        cot[j, i] = float("nan")
        exp = O.upscale_bwd(cot.numpy(), h, w, mode=0, dtype=np.float32)
        got = ops.upscale_bwd(cot.cuda(), h, w, None, 0)
        for a, b in zip(got, exp):
            assert np.array_equal(np.isnan(a.cpu().numpy()), np.isnan(b))
