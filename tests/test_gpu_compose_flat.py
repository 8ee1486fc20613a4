"""Compose without a resize takes its values in order: edges of its groups of
four, arrays off a 16-byte boundary, sizes past one wave of its CTAs.  The same
operations in the same order as the torch expression: bit for bit."""
import pytest
import torch

from lig_b200.levels import compose

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(1, 1), (1, 3), (5, 7), (33, 517), (1, 50001), (50001, 1), (2049, 2047)])
@pytest.mark.parametrize("off_render,off_prev", [(0, 0), (1, 1), (0, 2), (3, None), (0, None)])
def test_bit_identical(h, w, off_render, off_prev):
    g = torch.Generator(device="cuda").manual_seed(1)
    n = 3 * h * w

    def image(off):
        return (torch.rand(n + 4, generator=g, device="cuda") * 1.4 - 0.2)[off:off + n].view(h, w, 3)

    render = image(off_render)
    prev = None if off_prev is None else image(off_prev)
    lo, hi = torch.tensor(-0.25, device="cuda"), torch.tensor(1.125, device="cuda")
    est = torch.clamp(render, 0, 1) * (hi - lo) - 0.5 + lo
    exp = est if prev is None else prev + est
    assert torch.equal(compose(prev, render, lo, hi, False), exp)
    assert torch.equal(compose(prev, render, lo, hi, True), torch.clamp(exp, 0, 1))
