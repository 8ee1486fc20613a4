"""A batch of decodes (one projection and one forward launch): each image equals its single
render bit for bit, also where a view shows nothing of its set, a set has one
Gaussian, opacities below 1/255 leave phantom slots on a view's first Gaussian
(itself outside the view), covariance rows, and sets that are not fp32 rows."""
import pytest
import torch

from lig_b200.serve import GaussianSet, render_view, render_views
from tests._scene import chol_to_cov, scene

pytestmark = pytest.mark.gpu


def _set(n, side, seed, opac=None, cov=False, dtype=torch.float32):
    means, L, colors, op = scene(n, side, side, diag=(0.5, 4.0), seed=seed, opac=opac)
    return GaussianSet(means.to(dtype), (chol_to_cov(L) if cov else L).to(dtype),
                       colors.to(dtype), side, side, op, cholesky=not cov)


def test_views_equal_single_renders():
    big = _set(5000, 200, 1)
    dim = _set(3000, 150, 2, opac=(0.0, 0.02))   # many phantoms
    dim.means[0] = torch.tensor([-500.0, -500.0], device="cuda")
    views = [
        (big, 64, 80, (10.0, 20.0), (1.0, 1.0)),
        (dim, 70, 50, (0.0, 0.0), (0.5, 0.75)),
        (big, 33, 47, (1000.0, 1000.0), (1.0, 1.0)),    # shows nothing
        (_set(1, 20, 3), 20, 20, (0.0, 0.0), (1.0, 1.0)),
        (_set(700, 90, 4, cov=True), 120, 130, (5.0, 0.0), (2.0, 1.5)),
        (_set(900, 90, 5, opac=(0.2, 1.0)), 40, 41, (30.0, 30.0), (1.0, 1.0)),
    ]
    for got, (gs, h, w, o, s) in zip(render_views(views), views):
        assert torch.equal(got, render_view(gs, h, w, o, s)[0])
    without = [v for v in views if v[0].opacities is None]
    for got, (gs, h, w, o, s) in zip(render_views(without), without):
        assert torch.equal(got, render_view(gs, h, w, o, s)[0])


def test_views_of_double_sets_render_in_float():
    gs = _set(400, 80, 6, dtype=torch.float64)
    f = GaussianSet(gs.means.float(), gs.chol.float(), gs.rgbs.float(), 80, 80)
    got = render_views([(gs, 50, 60, (3.0, 4.0), (1.0, 1.0))])[0]
    assert torch.equal(got, render_view(f, 50, 60, (3.0, 4.0), (1.0, 1.0))[0])


def test_views_broadcast_colours_and_refuse_wrong_rows():
    gs = _set(300, 60, 7)
    flat = GaussianSet(gs.means, gs.chol, gs.rgbs[:1], 60, 60)
    wide = GaussianSet(gs.means, gs.chol, gs.rgbs[:1].expand(300, 3).contiguous(), 60, 60)
    v = (40, 50, (0.0, 0.0), (1.0, 1.0))
    assert torch.equal(render_views([(flat, *v)])[0], render_view(wide, *v)[0])
    with pytest.raises(RuntimeError):
        render_views([(GaussianSet(gs.means, gs.chol, gs.rgbs[:7], 60, 60), *v)])


@pytest.mark.parametrize("big", [False, True])
@pytest.mark.parametrize("block", [8, 16, 24])
def test_views_tile_sizes(block, big):
    h, w = (1100, 1205) if big else (129, 67)   # four pixels a lane from 4096 tiles on
    gs = _set(4000, 300, 8, opac=(0.3, 1.0) if big else None)
    args = (h, w, (7.0, 9.0), (2.0, 3.0))
    got = render_views([(gs, *args), (gs, 20, 30, (1.0, 1.0), (1.0, 1.0))], block)[0]
    assert torch.equal(got, render_view(gs, *args, block)[0])


@pytest.mark.parametrize("h,w", [(200, 30), (900, 900), (1990, 2010)])
def test_views_of_a_partly_visible_set(h, w):
    """From 2049 Gaussians on the counting kernels queue the visible ones: few,
    a fifth and all of the set, beside a small view of another set."""
    gs, other = _set(60000, 2048, 9), _set(2500, 100, 10)
    args = (h, w, (20.0, 31.0), (1.0, 1.0))
    got = render_views([(gs, *args), (other, 50, 60, (0.0, 0.0), (1.0, 1.0)), (gs, *args)])
    want = render_view(gs, *args)[0]
    assert torch.equal(got[0], want) and torch.equal(got[2], want)
