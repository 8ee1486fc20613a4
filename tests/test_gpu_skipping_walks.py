"""Values of the walks that skip pixels one by one (records without culling
data, large cotangents), with everything finite: the float sum backward with
opacities, and the gradient-aware forward and backward, against the library's
FP64 instantiation.

A large cotangent or colour would hide all other rows in one norm, so the rows
(pixels) that it enters and those that it does not are compared apart.
Tolerance (2-norm, relative): float rounding gives about 1e-6 a term; sigma of
an indefinite conic is good to about 1e-5 some twenty pixels out, and the sums
over its 500 pixels cancel to about a twentieth: 2e-4; 1e-3 allowed."""
import pytest
import torch

from lig_b200 import ops
from tests._scene import scene

pytestmark = pytest.mark.gpu

SIZES = [(61, 77, 16, 300), (50, 43, 8, 200), (47, 50, 12, 200)]
LARGE = [(1030, 1041, 16, 20000),   # 8x16 regions in the sum backward
         (1030, 1041, 16, 90000),   # 8x8
         (517, 515, 8, 9000)]


def _rows_agree(got, exp, apart):
    for rows in (apart, ~apart):
        assert rows.any()
        for a, b in zip(got, exp):
            if a is not None:
                a, b = a[rows].double(), b[rows]
                assert torch.isfinite(a).all() and torch.isfinite(b).all()
                assert (a - b).norm() <= 1e-3 * b.norm() and b.norm() > 0


def _run(H, W, B, n, opac, what, ga):
    """Forward planes and gradients in float and in double, and the Gaussians
    that the change touches (None: by the size of their colour gradients)."""
    means, L, colors, op = scene(n, H, W, diag=(0.5, 4.0), opac=opac, seed=n)
    xys, ext, con, cnt = ops.project_fwd(L, means, op, H, W, B, True)
    g = torch.Generator().manual_seed(12)
    cots = [torch.randn(H, W, 3, generator=g).cuda() for _ in range(4 if ga else 1)]
    cw = torch.randn(H, W, generator=g).cuda()
    some = torch.zeros(n, dtype=torch.bool, device="cuda")
    some[5::41] = True
    if what == "colour":
        colors[some, 1] = 2e8
    elif what == "conic":
        con[some, 1] = 1.5 * (con[some, 0] * con[some, 2]).sqrt()
    else:
        x, y = xys[5].round().long().tolist()
        cots[-1][min(max(y, 0), H - 1), min(max(x, 0), W - 1), 1] = 2e12
        some = None
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    res = []
    for dt in (torch.float32, torch.float64):
        a = (H, W, B, b.gaussian_ids_sorted, b.tile_bins, b.total,
             *[None if t is None else t.to(dt) for t in (xys, con, colors, op)])
        fwd = ops.raster_fwd(*a, ga)
        v = [t.to(dt) for t in cots]
        res.append((fwd[:5], ops.raster_bwd(*a, fwd[5], v[0], cw.to(dt), *v[1:])))
    return res, some


def _check_gradients(f, d, some):
    if some is None:  # the wild cotangent times an alpha of at least 1/255
        some = d[3].abs().amax(1) > 1e8
    names = ("v_xy", "v_abs", "v_con", "v_rgb", "v_op")
    assert len(f) == len(names)
    _rows_agree(f, d, some)


@pytest.mark.parametrize("what", ["cotangent", "colour", "conic"])
@pytest.mark.parametrize("H,W,B,n", SIZES + LARGE)
def test_sum_backward_with_opacities(H, W, B, n, what):
    ((_, f), (_, d)), some = _run(H, W, B, n, (0.4, 0.98), what, False)
    _check_gradients(f, d, some)


@pytest.mark.parametrize("what", ["cotangent", "colour", "conic"])
@pytest.mark.parametrize("opac", [None, (0.4, 0.98)])
@pytest.mark.parametrize("H,W,B,n", SIZES)
def test_gradient_aware(H, W, B, n, opac, what):
    ((pf, f), (pd, d)), some = _run(H, W, B, n, opac, what, True)
    if what == "colour":
        _rows_agree(pf, pd, pd[0].abs().amax(2) > 1e5)
    else:
        for a, b in zip(pf, pd):
            assert (a.double() - b).norm() <= 1e-3 * b.norm()
    # (a cotangent of the mixed derivative enters the colours' gradients through
    # the slopes: by their size all the same)
    _check_gradients(f, d, some)
