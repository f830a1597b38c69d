"""What the build takes for out of date: the extension belongs to one torch, an object to its own source and the headers."""

import os
import types

import pytest
import torch

from rbf_attention_b200 import _lib, build


def test_nothing_is_built_twice(built_library, monkeypatch):
    monkeypatch.setattr(build.subprocess, "run", lambda *a, **k: pytest.fail(f"built again: {a}"))
    assert build.build() == built_library


def test_another_torch_wants_another_extension(built_library, monkeypatch):
    commands = []

    def run(command, **kwargs):
        commands.append(command)
        return types.SimpleNamespace(returncode=1, stdout="", stderr="")

    monkeypatch.setattr(build.subprocess, "run", run)
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    with pytest.raises(RuntimeError, match="build failed"):
        build.build()
    assert len(commands) == 1 and build.HOST in commands[0] and '-DRBF_TORCH_VERSION="9.9.9"' in commands[0]
    monkeypatch.setattr(_lib, "_host", None)
    with pytest.raises(RuntimeError, match="built for torch .*, this is 9.9.9"):
        _lib.host()


@pytest.mark.parametrize("dep", ["HOST_SOURCE", "C_HEADER"])
def test_the_extension_follows_its_source_and_the_c_header(dep, built_library, monkeypatch, tmp_path):
    newer = tmp_path / "newer"
    newer.touch()
    later = os.path.getmtime(build.HOST) + 10
    os.utime(newer, (later, later))
    assert not build._host_stale()
    monkeypatch.setattr(build, dep, str(newer))
    assert build._host_stale()


def test_objects_depend_on_headers_and_not_on_one_another(built_library):
    names = {os.path.basename(h) for h in build._headers()}
    assert {"rbf_b200.h", "launch.h", "ptx.cuh", "common.cuh"} <= names
    assert not any(n.endswith((".o", ".cu", ".cpp")) for n in names)
