"""The pinned skip count of a BatchedFit that is dropped with steps in flight is
not handed out again before the device has written it."""
import gc

import pytest
import torch

from lig_b200.batch import BatchedFit

pytestmark = pytest.mark.gpu

SLEEP = 1_000_000_000  # SM cycles: about half a second


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("side", [False, True])
def test_skip_count_of_a_dropped_fit(graph, side):
    target = torch.rand(40, 48, 3, generator=torch.Generator().manual_seed(1)).cuda()
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        fit = BatchedFit([target], [60], graph=graph)
        for _ in range(4):  # captured from the third on
            fit.step()
        torch.cuda.synchronize()
        torch.cuda._sleep(SLEEP)
        fit.step()
    word = fit.host_skipped.data_ptr()
    del fit
    gc.collect()
    others = [torch.zeros(1, dtype=torch.int32, pin_memory=True) for _ in range(16)]
    assert not stream.query(), "the step must still be in flight"
    assert word not in [t.data_ptr() for t in others]
    torch.cuda.synchronize()
