"""Builds the test-only sources of tests/native with the library's own flags."""

import ctypes
import subprocess
from pathlib import Path

from gjxl_b200 import build

NATIVE = Path(__file__).resolve().parent / "native"


def load(name: str, directory: Path) -> ctypes.CDLL:
    """tests/native/<name>.cu as a shared library under `directory`."""
    library = directory / f"lib{name}.so"
    command = [build.NVCC, *build.ARCH, *build.COMMON, "-Xcompiler", "-fvisibility=default",
               "-shared", str(NATIVE / f"{name}.cu"), "-o", str(library), "-cudart", "shared"]
    result = subprocess.run(command, capture_output=True, text=True)
    assert result.returncode == 0, result.stderr
    return ctypes.CDLL(str(library))
