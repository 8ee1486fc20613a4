"""The binning's three routes — one CTA for small problems, shared-memory tile
counters, global atomics — give the same lists.  The emission-order outputs
(want_keys) keep the global-atomic route, so every size is binned both ways and
compared entry by entry, at the edges of the routes' rules."""
import pytest
import torch

from lig_b200 import ops
from tests._scene import scene

pytestmark = pytest.mark.gpu


def _compare(n, H, W, B, diag, opac=None):
    means, L, _, op = scene(n, H, W, diag=diag, opac=opac, seed=n % 97)
    xys, ext, _, cnt = ops.project_fwd(L, means, op, H, W, B, True)
    a = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B, want_keys=True)
    m = a.num_intersects
    assert m == b.num_intersects
    assert torch.equal(a.gaussian_ids_sorted[:m], b.gaussian_ids_sorted[:m])
    assert torch.equal(a.tile_bins, b.tile_bins)
    return xys, ext, cnt, a


@pytest.mark.parametrize("n,H,W,B,diag,opac", [
    (1, 20, 20, 16, (0.5, 3.0), None),
    (400, 64, 80, 16, (0.5, 4.0), (0.0, 1.0)),       # one CTA, phantom slots
    (2048, 16, 16, 16, (0.5, 2.0), None),            # one tile of more than 512 entries
    (2048, 512, 512, 16, (0.3, 0.6), None),          # 1024 tiles
    (2049, 512, 512, 16, (0.3, 0.6), None),          # shared counters
    (2048, 512, 528, 16, (0.3, 0.6), None),          # 1056 tiles
    (2000, 200, 200, 16, (6.0, 9.0), None),          # more than 8192 slots
    (70001, 700, 513, 16, (0.5, 6.0), (0.0, 1.0)),   # shared counters, phantom slots
    (30000, 384, 512, 2, (0.3, 1.5), None),          # 49152 tiles: the last shared size
    (30000, 386, 512, 2, (0.3, 1.5), None),          # 49408 tiles: global counters
    (2000003, 2048, 2048, 16, (0.3, 0.8), None),     # two CTAs per SM
])
def test_routes_agree(n, H, W, B, diag, opac):
    _compare(n, H, W, B, diag, opac)


@pytest.mark.parametrize("n,H,W", [(1500, 100, 120), (20000, 300, 300)])
def test_capacity_below_the_count_is_redone(n, H, W):
    xys, ext, cnt, a = _compare(n, H, W, 16, (0.5, 4.0))
    ops._CAP_HINT[ops._cap_key(n, H, W, 16, xys.device)] = 10
    b = ops.bin_gaussians(xys, ext, cnt, H, W, 16)
    m = a.num_intersects
    assert b.num_intersects == m and b.capacity >= m
    assert torch.equal(a.gaussian_ids_sorted[:m], b.gaussian_ids_sorted[:m])
    assert torch.equal(a.tile_bins, b.tile_bins)
