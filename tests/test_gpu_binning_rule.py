"""The binning gives the same lists on both sides of the rule that picks shared or
global tile counters: capacities one slot below and at its line (64 or a 160th
of the tiles a tile, 50 from two million Gaussians on), the last tile count of
the shared counters and the next.  Compared with the emission-order route."""
import pytest
import torch

from lig_b200 import _lib, ops
from tests._scene import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,H,W,B,diag,per_tile", [
    (5000, 512, 512, 16, (0.5, 4.0), 64),        # 1024 tiles
    (50000, 208, 816, 4, (0.3, 1.0), 66),        # 10608 tiles
    (100000, 256, 384, 2, (0.3, 0.8), 153),      # 24576 tiles
    (100000, 258, 384, 2, (0.3, 0.8), None),     # 24768: global counters whatever the slots
    (2000000, 512, 640, 4, (0.3, 0.5), 50),      # 20480 tiles
])
def test_both_sides_of_the_line(n, H, W, B, diag, per_tile):
    means, L, _, _ = scene(n, H, W, diag=diag, seed=n % 97)
    if n >= 2000000:
        means[: n - 100000] -= 5000.0  # most outside the image: few slots
    xys, ext, _, cnt = ops.project_fwd(L, means, None, H, W, B, True)
    ref = ops.bin_gaussians(xys, ext, cnt, H, W, B, want_keys=True)
    m, tiles = ref.num_intersects, -(-W // B) * -(-H // B)
    line = (per_tile or 400) * tiles
    assert 0 < m < line - 1
    need = [_lib.lib.lig_bin_workspace_bytes(n, c, tiles) for c in (line - 1, line)]
    assert (need[0] < need[1]) == (per_tile is not None)
    for cap in (m, line - 1, line):
        gids, bins = ops._run_bin(xys, ext, ref.cum_tiles_hit, ref.total, H, W, B, cap, False)[:2]
        assert torch.equal(gids[:m], ref.gaussian_ids_sorted[:m])
        assert torch.equal(bins, ref.tile_bins)
