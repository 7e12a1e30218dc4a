"""What build() makes, with the compilers replaced by a recorder: no compiler runs here."""
import os
import shutil
import types

import pytest

from tyr_b200 import build


@pytest.fixture
def recorder(monkeypatch, tmp_path):
    lib, calls = str(tmp_path / "libtyr_b200_attn.so"), str(tmp_path / "_calls.so")
    monkeypatch.setattr(build, "LIB_DIR", str(tmp_path))
    monkeypatch.setattr(build, "LIB_PATH", lib)
    monkeypatch.setattr(build, "CALLS_PATH", calls)
    ran = []

    def run(cmd, **kw):
        ran.append(os.path.basename(cmd[0]))
        open(cmd[cmd.index("-o") + 1], "w").close()
        return types.SimpleNamespace(returncode=0, stderr="", stdout="")

    monkeypatch.setattr(build.subprocess, "run", run)
    return ran


def test_library_and_calls_are_built_once(recorder):
    build.build()
    assert recorder == ["nvcc", "g++"] and not build.stale()
    build.build()
    assert recorder == ["nvcc", "g++"]
    build.build(force=True)
    assert recorder == ["nvcc", "g++"] * 2


def test_the_library_alone_needs_no_torch_and_no_host_compiler(recorder, monkeypatch):
    import torch
    monkeypatch.setattr(torch.version, "cuda", None)      # a CPU build of torch
    assert build.build() == build.LIB_PATH and recorder == ["nvcc"] and not build.stale()


def test_without_a_host_compiler(recorder, monkeypatch):
    which = shutil.which
    monkeypatch.setattr(build.shutil, "which", lambda n: None if n == "g++" else which(n))
    assert build.build() == build.LIB_PATH and recorder == ["nvcc"] and not build.stale()


def test_calls_are_stale_for_another_torch(recorder, monkeypatch):
    build.build()
    monkeypatch.setattr(build, "_calls_stamp", lambda: "another python and torch")
    assert build.stale() and not build.library_stale()
    build.build()
    assert recorder == ["nvcc", "g++", "g++"] and not build.stale()
