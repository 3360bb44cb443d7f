"""The module of the native calls belongs to one Python and one torch, follows its sources, and is optional (no GPU needed)."""
import os
import subprocess
import sysconfig
from pathlib import Path
from types import SimpleNamespace

import pytest
import torch

from hccl_b200 import _calls, build


@pytest.mark.skipif(torch.version.cuda is None, reason="a torch without CUDA")
def test_the_module_of_this_torch_is_there():
    assert _calls._module is not None
    assert Path(_calls._module.__file__) == build.torch_lib()


def test_another_torch_or_python_does_not_find_it(monkeypatch):
    ours = build.torch_lib()
    monkeypatch.setattr(torch, "__version__", "2.99.0")
    assert build.torch_lib() != ours and _calls._load() is None
    monkeypatch.undo()
    monkeypatch.setattr(sysconfig, "get_config_var", lambda name: "cpython-399-other")
    assert build.torch_lib() != ours and _calls._load() is None


@pytest.fixture
def compiler(monkeypatch, tmp_path):
    """Builds into a directory of its own with a compiler that writes an empty file; the commands it was given."""
    commands = []

    def run(cmd, **_):
        commands.append(cmd)
        Path(cmd[cmd.index("-o") + 1]).write_text("")
        return SimpleNamespace(returncode=0, stdout="", stderr="")

    monkeypatch.setattr(build, "LIB_DIR", tmp_path)
    monkeypatch.setattr(subprocess, "run", run)
    return commands


def test_it_is_built_again_when_a_header_of_the_c_api_or_its_source_changes(compiler, tmp_path):
    out = build.build_torch_calls()
    assert out.exists() and len(compiler) == 1
    build.build_torch_calls()
    assert len(compiler) == 1                                      # nothing has changed
    sources = [build.TORCH_SRC, *(build.CSRC / "include").rglob("*.h")]
    for src in (sources[0], max(sources, key=lambda p: p.stat().st_mtime)):
        os.utime(out, (src.stat().st_mtime - 1,) * 2)
        before = len(compiler)
        build.build_torch_calls()
        assert len(compiler) == before + 1
    other = tmp_path / "hccl_b200_torch.cpython-310-x86_64-linux-gnu.torch-1.0.so"
    other.write_text("")
    os.utime(other, (1, 1))
    build.build_torch_calls()
    assert not other.exists()                                      # it called a C API that has changed since


def test_a_failed_build_is_a_warning(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "LIB_DIR", tmp_path)
    monkeypatch.setattr(subprocess, "run", lambda *_, **__: SimpleNamespace(returncode=1, stdout="", stderr="no cuda_runtime.h"))
    with pytest.warns(UserWarning, match="cannot be compiled"):
        assert build.build_torch_calls() is None
    assert not list(tmp_path.iterdir())


def test_the_package_takes_the_modules_along():
    assert "hccl_b200_torch.*.so" in (build.ROOT / "build.sh").read_text()
