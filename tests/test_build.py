"""The native call path belongs to one torch, one Python and one set of argument structs (no GPU)."""
import ctypes as C
import os
import stat

import pytest


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A source folder whose nvcc and g++ are stand-ins that write an empty output file."""
    from tritonops_b200 import build
    csrc = tmp_path / "csrc"
    csrc.mkdir()
    tool = tmp_path / "tool"
    tool.write_text('#!/bin/sh\nwhile [ "$1" != -o ]; do shift; done\n: > "$2"\n')
    tool.chmod(tool.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setattr(build, "CSRC", str(csrc))
    monkeypatch.setattr(build, "LIB", str(csrc / "libb200attn.so"))
    monkeypatch.setenv("NVCC", str(tool))
    monkeypatch.setenv("CXX", str(tool))
    return build, csrc


def test_another_torch_needs_another_build(tree, monkeypatch):
    import torch
    build, csrc = tree
    build.build_library()
    assert not build._stale()
    first = build.host_path()
    assert os.path.exists(first)
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build._stale() and build.host_path() != first
    build.build_library()
    assert sorted(os.listdir(csrc)) == sorted(["libb200attn.so", os.path.basename(build.host_path())])


def test_a_failed_host_build_leaves_no_older_one_behind(tree, monkeypatch):
    build, csrc = tree
    build.build_library()
    monkeypatch.setenv("CXX", "false")
    with pytest.raises(RuntimeError):
        build.build_library(force=True)
    assert os.listdir(csrc) == ["libb200attn.so"] and build._stale()


def test_other_argument_structs_are_refused():
    from tritonops_b200 import _lib, build
    build.build_library()
    host = _lib.host()
    sizes = [C.sizeof(s) for s in _lib.HOST_STRUCTS]
    host.init(_lib.LIB_PATH, *sizes)
    for i in range(len(sizes)):
        with pytest.raises(RuntimeError):
            host.init(_lib.LIB_PATH, *sizes[:i], sizes[i] + 8, *sizes[i + 1:])
    with pytest.raises(RuntimeError):
        host.init(_lib.LIB_PATH, *sizes[:-1])
