"""A call that fails after the copy of its intersection count was enqueued waits
for that copy: the thread's pinned word is free for the next call (or the
thread's end)."""
import pytest
import torch

from lig_b200 import ops
from tests._scene import scene

pytestmark = pytest.mark.gpu

SLEEP = 1_000_000_000  # SM cycles: about half a second


def test_count_of_a_failed_call():
    H, W, n = 40, 48, 60
    means, L, colors, _ = scene(n, H, W)
    xys, ext, con, cnt = ops.project_fwd(L, means, None, H, W, 16, True)
    args = (xys, ext, cnt, con)
    b, _ = ops.bin_raster_fwd(*args, colors, None, H, W, 16, False)
    slot = ops._HostCount.slot()
    for call in (lambda: ops.bin_raster_fwd(*args, colors.cpu(), None, H, W, 16, False),
                 lambda: ops.bin_gaussians(xys, ext, cnt, H, W, 16,
                                           after_enqueue=lambda b: 1 / 0)):
        torch.cuda.synchronize()
        slot.fill_(-1)
        torch.cuda._sleep(SLEEP)
        with pytest.raises((RuntimeError, ZeroDivisionError)):
            call()
        assert int(slot) == b.num_intersects  # arrived before the call returned
