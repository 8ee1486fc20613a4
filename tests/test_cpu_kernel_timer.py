"""KernelTimer pairs the native operators' start and end events per thread."""
import threading

import torch

from lig_b200 import ops


class _Event:
    made = []

    def __init__(self, enable_timing=False):
        self.thread = threading.get_ident()
        _Event.made.append(self)

    def record(self, stream=None):
        self.recorded_at = len(_Event.made)


def test_two_threads_inside_one_timer(monkeypatch):
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    timer = ops.KernelTimer()
    with timer:
        timer._observe("begun before the timer", 1)
        timer._observe("here", 0)
        t = threading.Thread(target=lambda: (timer._observe("there", 0),
                                             started.set(), go_on.wait(10),
                                             timer._observe("there", 1)))
        started, go_on = threading.Event(), threading.Event()
        t.start()
        assert started.wait(10)
        timer._observe("here", 1)
        go_on.set()
        t.join()
    assert sorted(name for name, _, _ in timer.events) == ["here", "there"]
    for _, start, end in timer.events:
        assert start.thread == end.thread and start is not end
