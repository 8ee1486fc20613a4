"""The packed gradient-aware kernels (float) against the library's FP64
instantiation, which is held to the FP64 oracle elsewhere: tile sizes with and
without the packed backward, ragged images, short and long lists (1 to 8 lanes
a Gaussian, more than one batch), opacities, an optional wsum cotangent, and
the walk that skips pixels (non-finite records and cotangents).

Tolerance (2-norm, relative): float rounding gives about 1e-6.  A pixel whose
alpha lies within rounding of 1/255 may be decided differently in double: about
66 pixels per unit of sigma and Gaussian at a 5e-6 window, so at most a few of
the 64 x 80 pixels' terms, each 1/255 of a colour against a norm of about 40:
2e-4 a pixel for the planes, the same share of a gradient."""
import pytest
import torch

from lig_b200 import ops
from tests._scene import scene

pytestmark = pytest.mark.gpu

F64 = torch.float64


def _run(H, W, B, means, L, colors, op, cots, spoil=None):
    """Forward planes and gradients in float and in double on the float
    projection and tile lists."""
    xys, ext, con, cnt = ops.project_fwd(L, means, op, H, W, B, True)
    if spoil is not None:
        spoil(con, colors)
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    out = []
    for dt in (torch.float32, F64):
        c = [None if t is None else t.to(dt) for t in (xys, con, colors, op)]
        args = (H, W, B, b.gaussian_ids_sorted, b.tile_bins, b.total, *c)
        fwd = ops.raster_fwd(*args, True)
        v = [None if t is None else t.to(dt) for t in cots]
        # (a 32x32 tile's FP64 backward exceeds an SM's shared memory)
        bwd = ops.raster_bwd(*args, fwd[5], *v) if B <= 16 else []
        out.append(([t for t in fwd[:5]], [t for t in bwd if t is not None]))
    return out


def _cots(H, W, vw, seed=3):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    return [r(H, W, 3), r(H, W) if vw else None, r(H, W, 3), r(H, W, 3), r(H, W, 3)]


def _rel(a, b):
    return float((a.double() - b.double()).norm() / (b.double().norm() + 1e-30))


@pytest.mark.parametrize("H,W,B,n,opac,vw", [
    (64, 80, 16, 400, None, False),
    (61, 77, 16, 400, (0.05, 0.98), True),
    (48, 48, 16, 3, None, True),              # eight lanes a Gaussian
    (32, 32, 16, 1500, (0.05, 0.98), False),  # several batches a tile
    (50, 43, 8, 300, (0.05, 0.98), True),
    (40, 40, 8, 1200, None, False),
    (47, 50, 12, 300, (0.05, 0.98), True),
    (70, 66, 32, 300, None, True),
])
def test_packed_kernels_match_fp64(H, W, B, n, opac, vw):
    means, L, colors, op = scene(n, H, W, diag=(0.5, 4.0), opac=opac, seed=n)
    (f32, g32), (f64, g64) = _run(H, W, B, means, L, colors, op, _cots(H, W, vw))
    for a, b in zip(f32, f64):
        assert _rel(a, b) <= 1e-3
    for a, b in zip(g32, g64):
        assert _rel(a, b) <= 1e-3


@pytest.mark.parametrize("B", [16, 8])
def test_non_finite_values_stay_where_the_alpha_test_lets_them(B):
    """A NaN colour, a NaN conic, an indefinite conic and NaN / infinite
    cotangents spoil the same outputs as pixel-by-pixel skipping does."""
    H, W, n = 45, 52, 120
    means, L, colors, op = scene(n, H, W, diag=(0.5, 3.0), seed=9)

    def spoil(con, col):
        col[5, 1] = float("nan")
        con[11] = float("nan")
        con[17, 1] = 3 * con[17, 0]

    cots = _cots(H, W, True)
    cots[0][7, 9, 1] = float("nan")
    cots[3][30, 31, 2] = float("inf")
    cots[1][20, 3] = float("nan")
    (f32, g32), (f64, g64) = _run(H, W, B, means, L, colors, op, cots, spoil)
    for a, b in list(zip(f32, f64)) + list(zip(g32, g64)):
        assert torch.equal(torch.isnan(a), torch.isnan(b))
        ok = torch.isfinite(a) & torch.isfinite(b)
        assert ok.any()
