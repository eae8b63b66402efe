"""What the suite skips where the reference's sources are not there (CPU)."""
import os

import pytest

from oracle import ref_ffi
from tests import conftest


def _outcome(error):
    """What a test that raises `error` ends with."""
    hook = conftest.pytest_runtest_call(None)
    next(hook)
    try:
        hook.throw(error)
    except BaseException as e:  # (a skip is no Exception)
        return e
    return None


@pytest.mark.parametrize("there", [False, True])
def test_only_a_missing_adapter_is_skipped(monkeypatch, tmp_path, there):
    lib = tmp_path / "libdp3_adapter_check.so"
    if there:
        lib.write_bytes(b"no library")
    monkeypatch.setattr(conftest, "ADAPTER_LIB", str(lib))
    monkeypatch.setattr(ref_ffi, "REFERENCE", "")
    got = _outcome(OSError(f"{lib}: cannot open shared object file"))
    assert isinstance(got, OSError if there else pytest.skip.Exception)


def test_other_errors_are_not_skipped(monkeypatch):
    monkeypatch.setattr(ref_ffi, "REFERENCE", "")
    assert isinstance(_outcome(OSError("libother.so: undefined symbol")), OSError)
    assert isinstance(_outcome(ref_ffi.ReferenceMissing("no sources")), pytest.skip.Exception)
    assert os.path.basename(conftest.ADAPTER_LIB) == "libdp3_adapter_check.so"
