"""The float sum backward with opacities and / or a wsum cotangent on tiles of two
to five pixels, above and below the tile count from which taller regions are
taken, against the library's FP64 instantiation (tolerance as in the general
backward's other test)."""
import pytest
import torch

from lig_b200 import ops
from tests._scene import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(40, 47), (300, 330)])
@pytest.mark.parametrize("B", [2, 3, 4, 5])
@pytest.mark.parametrize("opac,vw", [((0.05, 0.98), False), ((0.05, 0.98), True), (None, True)])
def test_general_backward(H, W, B, opac, vw):
    n = H * W // 12
    means, L, colors, op = scene(n, H, W, diag=(0.5, 4.0), opac=opac, seed=B)
    xys, ext, con, cnt = ops.project_fwd(L, means, op, H, W, B, True)
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    g = torch.Generator().manual_seed(4)
    cot, cw = torch.randn(H, W, 3, generator=g).cuda(), torch.randn(H, W, generator=g).cuda()
    res = []
    for dt in (torch.float32, torch.float64):
        a = (H, W, B, b.gaussian_ids_sorted, b.tile_bins, b.total,
             *[None if t is None else t.to(dt) for t in (xys, con, colors, op)])
        fin = ops.raster_fwd(*a, False)[5]
        res.append(ops.raster_bwd(*a, fin, cot.to(dt), cw.to(dt) if vw else None))
    for got, exp in zip(*res):
        if got is not None:
            assert (got.double() - exp).norm() <= 1e-3 * exp.norm()
