"""The float gradient-aware forward at the tile sizes around which it changes its
regions (4 and 5, 16 to 21), against the library's FP64 instantiation (tolerance
as in the gradient-aware kernels' other test), with a record that has no culling
data."""
import pytest
import torch

from lig_b200 import ops
from tests._scene import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [2, 3, 4, 5, 16, 17, 20, 21])
@pytest.mark.parametrize("opac", [None, (0.05, 0.98)])
def test_forward(B, opac):
    n, H, W = 400, 61, 77
    means, L, colors, op = scene(n, H, W, diag=(0.5, 4.0), opac=opac, seed=B)
    xys, ext, con, cnt = ops.project_fwd(L, means, op, H, W, B, True)
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    colors[7, 1] = 3e8
    out = []
    for dt in (torch.float32, torch.float64):
        a = (H, W, B, b.gaussian_ids_sorted, b.tile_bins, b.total,
             *[None if t is None else t.to(dt) for t in (xys, con, colors, op)])
        out.append(ops.raster_fwd(*a, True))
    far = out[1][0][..., 1].abs() < 1e4  # pixels that Gaussian 7 does not reach
    assert far.any() and not far.all()
    for got, exp in zip(out[0][:5], out[1][:5]):
        for m in (far, ~far):
            assert (got[m].double() - exp[m]).norm() <= 1e-3 * exp[m].norm()
