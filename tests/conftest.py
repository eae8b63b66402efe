import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line(
        "markers", "gpu: needs a CUDA device (B200, sm_100a); run with -m gpu")


def _have_gpu():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if _have_gpu():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture(scope="session")
def built():
    """Builds the native libraries in-tree if they are missing or stale."""
    from dp3_b200 import build
    build.build_all()
    from oracle import oracle_ffi, ref_ffi
    oracle_ffi.build()
    if ref_ffi.available():
        ref_ffi.build()  # compiles only where the reference tree is present
    return True


ADAPTER_LIB = os.path.join(os.path.dirname(os.path.abspath(__file__)), "adapter", "_build",
                           "libdp3_adapter_check.so")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    """A test that compares with the reference's own solver is skipped where
    that library (or the adapter harness, built from the same sources) is
    neither built nor buildable (no reference sources)."""
    from oracle import ref_ffi
    try:
        return (yield)
    except ref_ffi.ReferenceMissing as e:
        pytest.skip(str(e))
    except OSError as e:
        # (a library that is there and does not load fails)
        if (ref_ffi.REFERENCE or os.path.basename(ADAPTER_LIB) not in str(e)
                or os.path.exists(ADAPTER_LIB)):
            raise
        pytest.skip(str(e))
