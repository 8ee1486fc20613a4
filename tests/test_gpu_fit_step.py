"""The fit engine's three fused calls against the separate entry points they
replace: gradients, loss, parameters, moments, step counts; the skipped step of
an overflowed binning; fp32 and 8-bit targets; the persistent walk; an image
without Gaussians; one and many loss chunks per image.

Both sides run the same arithmetic; gradients differ by the order of the
backward's float atomics (1e-6 of a gradient buffer's norm), and Adam's first
step divides by |g| + 1e-8."""
import pytest
import torch

from lig_b200 import _lib, ops
from lig_b200.batch import BatchedFit

pytestmark = pytest.mark.gpu

p = ops._p


def _fit(shapes, counts, u8, persistent):
    g = torch.Generator().manual_seed(11)
    targets = [torch.rand(h, w, 3, generator=g).cuda() for h, w in shapes]
    if u8:
        targets = [(t * 255).to(torch.uint8) for t in targets]
    return BatchedFit(targets, counts, persistent=persistent, graph=False)


def _separate_step(f):
    """One iteration through the separate entry points."""
    L, st = f.L, f._stream()
    f._bin(st)
    fwd = ("lig_raster_fwd_l2_u8_batch" if f.target.dtype == torch.uint8
           else "lig_raster_fwd_l2_batch")
    ops.call(fwd, _lib.LIG_F32, *L.args(), L.block, p(f.gids), p(f.bins), p(f.total), p(f.cum),
             p(f.xys), p(f.con), p(f.rgbs), None, p(f.target), 0, p(f.work), p(f.r_ws),
             f.r_ws.numel(), p(f.partials), p(f.img), None, p(f.loss), p(f.per_image), st)
    ops.call("lig_raster_bwd_diff_batch", _lib.LIG_F32, *L.args(), L.block, p(f.gids), p(f.bins),
             p(f.total), p(f.cum), p(f.xys), p(f.con), p(f.rgbs), None, None, p(f.img), p(f.one),
             0.0, 0, p(f.work), p(f.r_ws), f.r_ws.numel(), p(f.v_xy), p(f.v_abs), p(f.v_con),
             p(f.g_rgbs), None, st)
    ops.call("lig_project_bwd_batch", _lib.LIG_F32, *L.args(), 1, p(f.chol), p(f.means), None,
             L.block, p(f.v_xy), 2, p(f.v_con), 3, p(f.g_chol), p(f.g_means), st)
    ops.call("lig_adam_step_batch", L.n, L.args()[3], p(f.flat), p(f.grad), p(f.m), p(f.v), f.lr,
             f.b1, f.b2, f.eps, p(f.status), p(f.steps), p(f.skipped), p(f.adam_scratch),
             f.adam_scratch.numel(), st)


def _rel(a, b):
    return float((a.double() - b.double()).norm() / (b.double().norm() + 1e-30))


@pytest.mark.parametrize("shapes,counts,u8,persistent", [
    ([(61, 77)], [300], False, False),
    ([(61, 77), (40, 33), (130, 90)], [300, 0, 700], True, False),
    ([(61, 77), (40, 33), (130, 90)], [300, 0, 700], False, True),
    ([(1040, 1030)], [20000], True, False),     # 4290 tiles: several chunks, 8x16 regions
    ([(1040, 1030)], [90000], False, False),    # 8x8 regions
])
def test_fused_step_matches_separate_calls(shapes, counts, u8, persistent):
    a, b = _fit(shapes, counts, u8, persistent), _fit(shapes, counts, u8, False)
    for _ in range(3):
        b.flat.copy_(a.flat)  # lockstep: Adam's first steps amplify rounding
        b.m.copy_(a.m)
        b.v.copy_(a.v)
        a.step()
        _separate_step(b)
        torch.cuda.synchronize()
        assert torch.equal(a.cnt, b.cnt) and torch.equal(a.cum, b.cum)
        seen = a.cnt > 0
        assert torch.equal(a.xys[seen], b.xys[seen]) and torch.equal(a.ext[seen], b.ext[seen])
        assert torch.equal(a.bins, b.bins)
        assert torch.equal(a.gids[:int(a.total)], b.gids[:int(b.total)])
        assert torch.equal(a.img, b.img)
        assert torch.allclose(a.per_image, b.per_image, rtol=1e-6)
        assert torch.allclose(a.loss, b.loss, rtol=1e-6)
        assert _rel(a.grad, b.grad) <= 1e-5
        assert _rel(a.m, b.m) <= 1e-5 and _rel(a.v, b.v) <= 1e-5
        assert _rel(a.flat, b.flat) <= 1e-6
        assert torch.equal(a.steps, b.steps)
    assert int(a.host_skipped[0]) == 0


def test_overflowed_step_updates_nothing_and_is_counted():
    f = _fit([(61, 77), (50, 50)], [300, 200], False, False)
    f._size_capacity(0)  # 4096 slots
    f.gids = f.gids[:64]
    f.capacity = 64
    before = f.flat.clone(), f.m.clone(), f.v.clone()
    f.step()
    torch.cuda.synchronize()
    assert int(f.skipped) == 1 and int(f.host_skipped[0]) == 1
    assert f.steps.tolist() == [0, 0]
    assert all(torch.equal(x, y) for x, y in zip(before, (f.flat, f.m, f.v)))
