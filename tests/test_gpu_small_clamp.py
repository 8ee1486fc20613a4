"""A backward clamp below 1/255: the alpha rule min(clamp, exp(-sigma)) < 1/255
then skips every pixel, so every gradient is zero — with and without opacities,
in float and in double, in every walk.  Just above 1/255 the float gradients are
the double ones (tolerance as in the general backward's test)."""
import pytest
import torch

from lig_b200 import ops
from tests._scene import scene

pytestmark = pytest.mark.gpu


def _gradients(H, W, B, n, opac, clamp, dt):
    means, L, colors, op = scene(n, H, W, diag=(0.5, 4.0), opac=opac, seed=n)
    xys, ext, con, cnt = ops.project_fwd(L, means, op, H, W, B, True)
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    a = (H, W, B, b.gaussian_ids_sorted, b.tile_bins, b.total,
         *[None if t is None else t.to(dt) for t in (xys, con, colors, op)])
    g = torch.Generator().manual_seed(8)
    v = [torch.randn(H, W, 3, generator=g).to("cuda", dt) for _ in range(4)]
    fin = ops.raster_fwd(*a, False)[5]
    out = [*ops.raster_bwd(*a, fin, v[0], None, alpha_clamp=clamp)]
    one = torch.ones((), dtype=dt, device="cuda")
    out += ops.raster_bwd_diff(*a, fin, v[0], one, alpha_clamp=clamp)
    out += ops.raster_bwd(*a, fin, v[0], None, *v[1:], alpha_clamp=clamp)
    return [t for t in out if t is not None]


@pytest.mark.parametrize("H,W,B,n", [(61, 77, 16, 300), (50, 43, 8, 200), (47, 50, 12, 200),
                                     (1030, 1041, 16, 20000),   # 8x16 regions
                                     (1030, 1041, 16, 90000)])  # 8x8 regions
@pytest.mark.parametrize("opac", [None, (0.4, 0.98)])
def test_clamp_around_one_over_255(H, W, B, n, opac):
    assert all((t == 0).all() for t in _gradients(H, W, B, n, opac, 0.003, torch.float32))
    if n <= 300:
        assert all((t == 0).all() for t in _gradients(H, W, B, n, opac, 0.003, torch.float64))
    got = _gradients(H, W, B, n, opac, 0.004, torch.float32)
    exp = _gradients(H, W, B, n, opac, 0.004, torch.float64)
    # (the fit's backward without opacities leaves v_xy_abs zero)
    assert sum(bool(b.norm() > 0) for b in exp) >= len(exp) - 1
    for a, b in zip(got, exp):
        assert (a.double() - b).norm() <= 1e-3 * b.norm()
