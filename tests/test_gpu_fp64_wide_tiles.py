"""FP64 sum forward, plain and with the loss fused in, on tiles wider than 16 at
small tile counts: from 25 on a CTA's records fill 48 KB, the most a kernel is
given without asking, and the kernel's own shared words come on top.  Against
the dense FP64 oracle, tolerance as for the other tile sizes."""
import numpy as np
import pytest
import torch

from lig_b200 import _lib, ops
from oracle import oracle as O
from tests._scene import np_, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [17, 24, 25, 29, 32])
@pytest.mark.parametrize("opac", [None, (0.1, 0.99)])
def test_sum_forward(B, opac):
    n, H, W = 250, 70, 83
    means, L, colors, op = scene(n, H, W, diag=(0.5, 4.0), opac=opac, dtype=torch.float64)
    xys, ext, con, cnt = ops.project_fwd(L, means, op, H, W, B, True)
    b = ops.bin_gaussians(xys, ext, cnt, H, W, B)
    a = (H, W, B, b.gaussian_ids_sorted, b.tile_bins, b.total, xys, con, colors, op)
    d = O.dense_fwd_f64(H, W, B, np_(xys), np_(ext), np_(cnt), np_(con), np_(colors), np_(op))
    img, wsum = ops.raster_fwd(*a, False)[:2]
    assert np.abs(np_(img) - d["img"]).max() <= 1e-9
    assert np.abs(np_(wsum) - d["wsum"]).max() <= 1e-9
    target = torch.rand(H, W, 3, generator=torch.Generator().manual_seed(1),
                        dtype=torch.float64).cuda()
    diff, _, loss = ops.raster_fwd_l2(*a, target)
    x, t = d["img"], np_(target)
    err = np.clip(x, 0, 1) - t
    assert np.abs(np_(diff) - np.where((x >= 0) & (x <= 1), err, 0)).max() <= 1e-9
    assert abs(float(loss) - np.mean(err ** 2)) <= 1e-9
    # the persistent walk of the same tiles
    i32 = lambda v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    hs, ws, ns = i32([H]), i32([W]), i32([n])
    rws = torch.empty(_lib.lib.lig_raster_workspace_bytes(_lib.LIG_F64, n), dtype=torch.uint8,
                      device="cuda")
    work = torch.zeros(1, dtype=torch.int32, device="cuda")
    img2, wsum2, fin2 = torch.empty_like(img), torch.empty_like(wsum), i32([0] * H * W).cuda()
    p = ops._p
    ops.call("lig_raster_fwd_batch", _lib.LIG_F64, 1, p(hs), p(ws), p(ns), B,
             p(b.gaussian_ids_sorted), p(b.tile_bins), p(b.total), p(b.cum_tiles_hit), p(xys),
             p(con), p(colors), p(op), 1, p(work), p(rws), rws.numel(), p(img2), p(wsum2), None,
             None, None, p(fin2), ops._stream(img.device))
    assert torch.equal(img2, img) and torch.equal(wsum2, wsum)
