"""What an import says when a built file is missing or is another torch's."""

import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest
import torch

PACKAGE = Path(__file__).resolve().parent.parent / "tessiq_b200"


def message_of_import(tmp_path, with_library):
    copy = tmp_path / "tessiq_b200"
    copy.mkdir()
    for source in PACKAGE.glob("*.py"):
        shutil.copy(source, copy)
    if with_library:
        os.symlink(PACKAGE / "libtessiq_b200.so", copy / "libtessiq_b200.so")
    result = subprocess.run([sys.executable, "-c", "import tessiq_b200.ops"], cwd=tmp_path, capture_output=True, text=True,
                            env={**os.environ, "PYTHONPATH": str(tmp_path)})
    assert result.returncode != 0
    return result.stderr


@pytest.mark.parametrize("with_library, missing", [(False, "libtessiq_b200.so"), (True, "_launcher.so")])
def test_a_missing_file_is_named_with_the_command_that_builds_it(tmp_path, with_library, missing):
    message = message_of_import(tmp_path, with_library)
    assert f"{missing} is missing" in message and "python -m tessiq_b200.build" in message


def test_the_launcher_is_loaded_into_its_own_torch_only(monkeypatch):
    from tessiq_b200 import _lib

    assert _lib.load_launcher().BUILT_FOR.startswith(f"torch {torch.__version__}")
    monkeypatch.setattr(torch, "__version__", "2.99.0+cu999")
    with pytest.raises(ImportError, match="built for torch .*python -m tessiq_b200.build"):
        _lib.load_launcher()


def test_the_launcher_is_built_again_for_another_torch(monkeypatch, tmp_path):
    from tessiq_b200 import build

    running = f"torch {torch.__version__}, Python {sys.version_info.major}.{sys.version_info.minor}"
    monkeypatch.setattr(build, "LAUNCHER", tmp_path / "_launcher.so")
    monkeypatch.setattr(build, "OBJECTS", tmp_path)
    assert not build.launcher_is_current(running)
    build.LAUNCHER.touch()      # newer than every source
    assert not build.launcher_is_current(running)
    (tmp_path / "launcher.built_for").write_text(running)
    assert build.launcher_is_current(running)
    assert not build.launcher_is_current(running.replace("torch ", "torch 2.99."))
    os.utime(build.LAUNCHER, (0, 0))
    assert not build.launcher_is_current(running)
