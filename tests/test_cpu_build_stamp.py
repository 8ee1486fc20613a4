"""The native half of ops.py is rebuilt when what it was built against changes,
torch's version above all, and not otherwise."""
import os

import pytest

from lig_b200 import build


@pytest.fixture
def host(tmp_path, monkeypatch):
    """build._build_host on a folder of its own, counting the builds."""
    src, lib = tmp_path / "host.cpp", tmp_path / "_host.so"
    src.write_text("")
    monkeypatch.setattr(build, "HOST_SRC", str(src))
    monkeypatch.setattr(build, "HOST_LIB", str(lib))
    monkeypatch.setattr(build, "HOST_STAMP", str(tmp_path / "host.stamp"))
    built = []
    monkeypatch.setattr(build, "_run_host", lambda cmd: (built.append(cmd), lib.write_text("")))
    return built


def test_same_command_is_not_repeated(host):
    build._build_host()
    build._build_host()
    assert len(host) == 1


def test_another_torch_rebuilds(host, monkeypatch):
    import torch
    build._build_host()
    monkeypatch.setattr(torch, "__version__", "0.0.1+other")
    build._build_host()
    assert len(host) == 2


def test_newer_source_or_lost_library_rebuilds(host):
    build._build_host()
    later = os.path.getmtime(build.HOST_LIB) + 10
    os.utime(build.HOST_SRC, (later, later))
    build._build_host()
    assert len(host) == 2
    os.remove(build.HOST_LIB)
    build._build_host()
    assert len(host) == 3
