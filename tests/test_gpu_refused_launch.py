"""A launch that needs more shared memory than an SM has is refused with an error,
and leaves none behind for the program's next call."""
import pytest
import torch

from lig_b200 import _lib, ops
from tests._scene import scene

pytestmark = pytest.mark.gpu


def test_error_is_reported_once():
    H, W, B, n = 40, 50, 32, 30
    means, L, colors, _ = scene(n, H, W, dtype=torch.float64)
    xys, ext, con, cnt = ops.project_fwd(L, means, None, H, W, B, True)
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    a = (H, W, B, b.gaussian_ids_sorted, b.tile_bins, b.total, xys, con, colors, None)
    fin = torch.zeros(H, W, dtype=torch.int32, device="cuda")
    with pytest.raises(_lib.LigError):
        ops.raster_bwd(*a, fin, torch.ones(H, W, 3, dtype=torch.float64, device="cuda"), None)
    assert float((torch.zeros(4, device="cuda") + 1).sum()) == 4  # torch checks its launch
