"""lig_level_compose on rows so long that sixteen of them exceed 4 GiB: without a
resize the sums are those of the torch expression, bit for bit."""
import pytest
import torch

from lig_b200.levels import compose

pytestmark = pytest.mark.gpu

LO, HI = -0.25, 1.125


def _est(render):
    return torch.clamp(render, 0, 1) * (HI - LO) - 0.5 + LO


@pytest.mark.parametrize("same_size_prev", [False, True])
def test_rows_beyond_32_bit_offsets(same_size_prev):
    H, W = 17, 22_369_632  # 16 rows: 4 GiB and 1 KiB
    render = torch.rand(H, W, 3, device="cuda")
    prev = torch.rand(H, W, 3, device="cuda") if same_size_prev else None
    out = compose(prev, render, LO, HI, False)
    for r in range(H):
        base = prev[r] if same_size_prev else 0
        assert torch.equal(out[r], base + _est(render[r]))
