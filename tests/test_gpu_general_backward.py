"""The float sum backward with opacities and / or a wsum cotangent (packed pair
walk) against the library's FP64 instantiation, which is held to the FP64
oracle elsewhere: the three region heights (by tile count and density), other
tile sizes, ragged images, the explicit and the fused-loss cotangents, and the
walk that skips pixels (non-finite records and cotangents).

Tolerance (2-norm, relative): float rounding gives about 1e-6; a pixel whose
alpha lies within rounding of 1/255 may be decided differently in double, which
moves a gradient by 1/255 of one of its hundreds of terms: 1e-3."""
import pytest
import torch

from lig_b200 import ops
from tests._scene import scene

pytestmark = pytest.mark.gpu


def _setup(H, W, B, n, opac, spoil=None):
    means, L, colors, op = scene(n, H, W, diag=(0.5, 4.0), opac=opac, seed=n)
    xys, ext, con, cnt = ops.project_fwd(L, means, op, H, W, B, True)
    if spoil is not None:
        spoil(con, colors)
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    lists = (b.gaussian_ids_sorted, b.tile_bins, b.total)

    def args(dt):
        return (H, W, B, *lists, *[None if t is None else t.to(dt)
                                   for t in (xys, con, colors, op)])
    return args


def _rel(a, b):
    return float((a.double() - b.double()).norm() / (b.double().norm() + 1e-30))


def _check(got, exp, tol=1e-3):
    for a, b in zip(got, exp):
        if a is not None:
            assert _rel(a, b) <= tol


@pytest.mark.parametrize("H,W,B,n,opac,vw", [
    (61, 77, 16, 400, (0.05, 0.98), True),
    (64, 48, 16, 3, (0.05, 0.98), False),            # eight lanes a Gaussian
    (32, 32, 16, 1500, None, True),                  # several batches a tile
    (47, 50, 12, 300, (0.05, 0.98), True),
    (1030, 1041, 16, 20000, (0.05, 0.98), True),     # 8x16 regions
    (1030, 1041, 16, 90000, (0.05, 0.98), False),    # 8x8 regions
    (517, 515, 8, 9000, (0.05, 0.98), True),         # 8x8 tiles
])
def test_general_walk_matches_fp64(H, W, B, n, opac, vw):
    args = _setup(H, W, B, n, opac)
    g = torch.Generator().manual_seed(4)
    cot = torch.randn(H, W, 3, generator=g).cuda()
    cw = torch.randn(H, W, generator=g).cuda() if vw else None
    res = []
    for dt in (torch.float32, torch.float64):
        a = args(dt)
        fin = ops.raster_fwd(*a, False)[5]
        res.append(ops.raster_bwd(*a, fin, cot.to(dt), None if cw is None else cw.to(dt)))
    _check(*res)


def test_fused_loss_backward_with_opacities_matches_fp64():
    H, W, B, n = 90, 70, 16, 500
    args = _setup(H, W, B, n, (0.05, 0.98))
    target = torch.rand(H, W, 3, generator=torch.Generator().manual_seed(5)).cuda()
    res = []
    for dt in (torch.float32, torch.float64):
        a, t = args(dt), target.to(dt)
        gl = torch.tensor(1.3, dtype=dt, device="cuda")
        diff, fin, _ = ops.raster_fwd_l2(*a, t)
        img, _, _, _, _, fin2 = ops.raster_fwd(*a, False)
        res.append(ops.raster_bwd_diff(*a, fin, diff, gl)
                   + ops.raster_bwd_l2(*a, fin2, img, t, gl))
    _check(*res)


@pytest.mark.parametrize("H,W,B,n", [(45, 52, 16, 120), (530, 520, 8, 6000)])
def test_non_finite_values_stay_where_the_alpha_test_lets_them(H, W, B, n):
    def spoil(con, col):
        col[5, 1] = float("nan")
        con[11] = float("nan")
        con[17, 1] = 3 * con[17, 0]

    args = _setup(H, W, B, n, (0.3, 0.98), spoil)
    g = torch.Generator().manual_seed(6)
    cot, cw = torch.randn(H, W, 3, generator=g).cuda(), torch.randn(H, W, generator=g).cuda()
    cot[7, 9, 1] = float("nan")
    cw[20, 3] = float("inf")
    res = []
    for dt in (torch.float32, torch.float64):
        a = args(dt)
        fin = ops.raster_fwd(*a, False)[5]
        res.append(ops.raster_bwd(*a, fin, cot.to(dt), cw.to(dt)))
    for a, b in zip(*res):
        assert torch.equal(torch.isnan(a), torch.isnan(b))
        assert (torch.isfinite(a) & torch.isfinite(b)).any()


@pytest.mark.parametrize("H,W,B,n", [(61, 77, 16, 300), (1030, 1041, 16, 20000),
                                     (1030, 1041, 16, 90000), (517, 515, 8, 9000)])
def test_lean_walk_with_records_without_culling_data(H, W, B, n):
    """Without opacities a warp's round takes the alpha cut's compare or, with an
    indefinite or nearly degenerate conic among its Gaussians, the float test."""
    def spoil(con, col):
        con[5::41, 1] = 1.2 * con[5::41, 0]                       # indefinite
        con[7::53, 1] = (0.9996 * con[7::53, 0] * con[7::53, 2]).sqrt()

    args = _setup(H, W, B, n, None, spoil)
    cot = torch.randn(H, W, 3, generator=torch.Generator().manual_seed(7)).cuda()
    res = []
    for dt in (torch.float32, torch.float64):
        a = args(dt)
        fin = ops.raster_fwd(*a, False)[5]
        res.append(ops.raster_bwd(*a, fin, cot.to(dt), None))
    # the degenerate records' own sums reach far and cancel: held apart
    ok = torch.ones(n, dtype=torch.bool, device="cuda")
    ok[5::41] = ok[7::53] = False
    _check([t[ok] for t in res[0] if t is not None], [t[ok] for t in res[1] if t is not None])
    assert all(torch.isfinite(t).all() for t in res[0] if t is not None)
