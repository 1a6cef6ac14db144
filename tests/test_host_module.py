"""The native host module is an accelerator of the launches, not a condition for them."""
import platform

import pytest

from mlperf_training_b200.csrc import build
from mlperf_training_b200.ops import _lib


def test_kernel_library_is_built_without_the_host_module(monkeypatch, tmp_path, capsys):
    """A machine on which the module does not compile gets the kernel library, and no module of an older build beside it."""
    def fails(force=False):
        raise RuntimeError("g++ failed for host.cpp")
    lib = tmp_path / "lib.so"
    lib.touch()
    (tmp_path / build.HOST_LIB_NAME).touch()
    for name, value in (("build_host", fails), ("sources", lambda: []), ("LIB_PATH", lib), ("PKG", tmp_path), ("CSRC", tmp_path),
                        ("_nvcc", lambda: "nvcc")):
        monkeypatch.setattr(build, name, value)
    assert build.build() == lib
    assert not (tmp_path / build.HOST_LIB_NAME).exists() and "g++ failed" in capsys.readouterr().err


@pytest.mark.parametrize("content", [b"", b"\x7fELF cut short"])
def test_a_module_that_does_not_load_is_passed_by(monkeypatch, tmp_path, content):
    path = tmp_path / build.HOST_LIB_NAME
    path.write_bytes(content)
    monkeypatch.setattr(_lib, "HOST_PATH", path)
    with pytest.warns(RuntimeWarning, match="does not load"):
        assert _lib._import_host() is None


def test_the_built_module_loads():
    if platform.machine() != "x86_64" or not _lib.HOST_PATH.exists():
        pytest.skip("no module here")
    assert _lib.host is not None and _lib.call is _lib.host.call
