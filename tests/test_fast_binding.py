"""The operators past ctypes: an extension that is missing is compiled, and one that cannot be compiled or loaded leaves ctypes."""
import subprocess

import pytest


@pytest.fixture
def elsewhere(pkg, tmp_path, monkeypatch):
    """The extension's place moved to an empty folder, and nothing loaded yet."""
    pkg.build.build_library()
    monkeypatch.setattr(pkg.build, "FAST_PATH", tmp_path / pkg.build.FAST_PATH.name)
    monkeypatch.setattr(pkg.capi, "_FAST", None)
    stamp = pkg.build.BUILD_DIR / (pkg.build.FAST_PATH.name + ".txt")
    was = stamp.read_text() if stamp.exists() else None
    yield pkg.build.FAST_PATH
    if was is not None:
        stamp.write_text(was)


def has_headers(pkg):
    return (pkg.build.Path(pkg.build.sysconfig.get_paths()["include"]) / "Python.h").exists()


def test_a_missing_extension_is_compiled_beside_a_current_library(pkg, elsewhere):
    if not has_headers(pkg):
        pytest.skip("no CPython headers")
    before = pkg.build.LIB_PATH.stat().st_mtime_ns
    pkg.build.build_library()
    assert elsewhere.exists() and pkg.build.LIB_PATH.stat().st_mtime_ns == before
    at = elsewhere.stat().st_mtime_ns
    pkg.build.build_library()
    assert elsewhere.stat().st_mtime_ns == at  # and once only
    assert not isinstance(pkg.capi.fast(), pkg.capi._ThroughCtypes)


@pytest.mark.parametrize("how", ["compiler says no", "no compiler"])
def test_a_compiler_that_fails_leaves_the_library_usable(pkg, elsewhere, monkeypatch, how):
    if not has_headers(pkg):
        pytest.skip("no CPython headers")

    def run(cmd, **kw):
        if how == "no compiler":
            raise FileNotFoundError(cmd[0])
        return subprocess.CompletedProcess(cmd, 1, "", "error: no")

    monkeypatch.setattr(pkg.build.subprocess, "run", run)
    with pytest.warns(UserWarning, match="ctypes"):
        assert pkg.build.build_library() == pkg.build.LIB_PATH
    assert not elsewhere.exists()
    assert pkg.capi.fast().softmax(0, 0, 1, 1, 0, 0, 0) is None


def test_a_file_that_cannot_be_loaded_leaves_ctypes(pkg, elsewhere):
    elsewhere.write_bytes(b"not a library")
    with pytest.warns(UserWarning, match="ctypes"):
        assert pkg.capi.fast().gemm() is None
    assert isinstance(pkg.capi.fast(), pkg.capi._ThroughCtypes)
