import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: long-running")


@pytest.hookimpl(trylast=True)
def pytest_collection_modifyitems(items):
    """Where the reference's kernels are not built (its sources are absent), the
    modules that compare with them fail: they run last, so that a run which
    stops at its first failure has run everything else."""
    from oracle import ref

    if not os.path.exists(ref.LIB_PATH):
        items.sort(key=lambda item: getattr(item.module, "ref", None) is ref)
