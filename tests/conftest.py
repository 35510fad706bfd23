import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


BINDING = ROOT / "integration" / "_build" / "libgjxl_b200_encoder.so"


def _skip_without_reference(outcome):
    """A test that ends at the oracle's library, the reference's CUDA path or the
    encoder binding being absent is skipped: all are built from the reference's
    sources. Built, but not loading, they fail the test as ever."""
    if outcome.excinfo is None:
        return
    from oracle import ref
    if ref.available():
        return
    error = outcome.excinfo[1]
    if isinstance(error, ref.LibraryMissing):
        missing = ref.LIBRARY_PATH
    else:
        missing = next((p for p in (BINDING, ref.CUDA_LIBRARY_PATH)
                        if p.name in str(error) and not p.exists()), None)
    if missing is not None:
        outcome.force_exception(pytest.skip.Exception(f"{missing.name} is not built"))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_setup(item):
    _skip_without_reference((yield))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    _skip_without_reference((yield))


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gjxl_b200 import _lib
    _lib.load()
    return torch.device("cuda:0")
