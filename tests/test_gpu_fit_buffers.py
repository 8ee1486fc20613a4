"""A BatchedFit holds no gradient rows that its step does not use."""
import pytest
import torch

from lig_b200.batch import BatchedFit

pytestmark = pytest.mark.gpu


def test_separate_gradient_rows_on_demand():
    fit = BatchedFit([torch.rand(40, 48, 3, device="cuda")], [60])
    for _ in range(4):
        fit.step()
    fit.render()
    torch.cuda.synchronize()
    assert not {"v_xy", "v_abs", "v_con"} & set(vars(fit))
    assert fit.v_xy.shape == fit.v_abs.shape == (60, 2) and fit.v_con.shape == (60, 3)
    assert fit.v_xy is fit.v_xy
