"""What an import says when a built file is missing."""

import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

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
