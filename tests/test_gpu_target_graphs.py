"""BatchedFit.step(target) with a float32 and a uint8 target at one address: each
takes its own captured graph.  Both views lie in one allocation, so either
reading stays inside it."""
import pytest
import torch

from lig_b200.batch import BatchedFit

pytestmark = pytest.mark.gpu


def test_float_and_byte_targets_at_one_address():
    h, w, n = 40, 48, 60
    buf = torch.rand(3 * h * w, generator=torch.Generator().manual_seed(2)).cuda()
    targets = [buf.view(h * w, 3), buf.view(torch.uint8)[:3 * h * w].view(h * w, 3)]
    assert targets[0].data_ptr() == targets[1].data_ptr()
    a, b = (BatchedFit([buf.view(h, w, 3)], [n], graph=g) for g in (True, False))
    for k in (0, 0, 0, 1, 0, 1, 1, 0):
        b.flat.copy_(a.flat)
        b.m.copy_(a.m)
        b.v.copy_(a.v)
        a.step(targets[k])
        b.step(targets[k])
        torch.cuda.synchronize()
        assert torch.equal(a.img, b.img)
        assert torch.allclose(a.loss, b.loss, rtol=1e-6)
