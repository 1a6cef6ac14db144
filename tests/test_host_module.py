"""The native host module is an accelerator of the launches, not a condition for them."""
from mlperf_training_b200.csrc import build


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
