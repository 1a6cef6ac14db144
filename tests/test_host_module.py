"""The native host module is an accelerator of the launches, not a condition for them."""
import ctypes
import platform

import pytest
import torch

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


GATE = [None, 2560, None, None, None, None, None, None, 7, 512, 1e-6]      # b200_hstu_gate_cat_fwd up to its rate
CALLS = [
    # each is refused before anything is launched, and says what it was given
    ("b200_norm_fwd", [1, None, None, None, None, None, None, None, None, 5, 7, 1e-5, 0, None], RuntimeError, "code 300.*D=7 "),
    ("b200_norm_fwd", [True, 0, 0, 0, 0, 0, 0, 0, 0, 5, 2 ** 32 + 9, 1, False, 0], RuntimeError, "D=9 "),      # an int wraps
    ("b200_norm_fwd", [0, None, None, None, None, None, None, None, None, 5, -3, 1e-5, 0, None], RuntimeError, "D=-3 "),
    ("b200_cross_entropy", [None, None, None, None, 3, 2 ** 40 + 1, 16, 1.0, 1, -100, None], RuntimeError, "pitch 1099511627777 "),
    ("b200_hstu_gate_cat_fwd", GATE + [1.5, 2 ** 64 - 1, None], RuntimeError, "rate 1.500000 "),
    ("b200_hstu_gate_cat_fwd", GATE + [3, 0, None], RuntimeError, "rate 3.000000 "),                            # an int for a float
    ("b200_hstu_gate_cat_fwd", GATE + [float("nan"), 0, None], RuntimeError, "rate -?nan "),
    ("b200_norm_fwd", [1, None], TypeError, None),                                                                # too few
    ("b200_norm_fwd", [1, None, None, None, None, None, None, None, None, 5, "7", 1e-5, 0, None], ctypes.ArgumentError, None),
    ("b200_norm_fwd", [1, None, None, None, None, None, None, None, None, 5, 7, torch.tensor(1e-5), 0, None], RuntimeError, "code 300"),
    ("b200_cross_entropy", [None, None, None, None, 3, 2 ** 64 + 5, 16, 1.0, 1, -100, None], RuntimeError, "pitch 5 "),
    ("b200_no_such_launcher", [1], AttributeError, None),
]


@pytest.mark.parametrize("name,args,error,text", CALLS)
def test_calls_are_converted_as_by_ctypes(name, args, error, text):
    _lib.load()
    told = []
    for call in (_lib._call_ctypes, _lib.call):
        with pytest.raises(error, match=text) as e:
            call(name, *args)
        told.append(str(e.value))
    assert told[0] == told[1]


def test_pointer_arrays_pass_through():
    _lib.load()
    for call in (_lib._call_ctypes, _lib.call):
        out = (ctypes.c_longlong * 2)()
        call("b200_attn_bwd_plan", 1, 2000, 2000, 64, 8, 64, 1, 0, out)
        assert out[0] > 0 and out[1] > 0
