"""The extension module that calls the C ABI (csrc/py_calls.cc) against ctypes; entry points that refuse their arguments return
before they touch a device."""
import ctypes

import numpy as np
import pytest

from scirust_b200 import _build
from scirust_b200.ops import _lib
from scirust_b200.parallel import symm  # noqa: F401  (declares the entry points that take references)


@pytest.fixture(scope="module")
def calls():
    _lib.cuda()
    got = _lib._native_calls()
    if not got:
        pytest.skip("built without the Python headers")
    return got


def test_every_entry_point_is_there(calls):
    import re
    assert set(calls) == {re.search(r"(sb_\w+)\(", d).group(1) for _, d in _build.cuda_entry_points()}


def test_arguments_and_results_are_those_of_ctypes(calls):
    lib = _lib.cuda()
    for name, args in (("sb_swiglu_fwd", (None, None, 0, 0, None)),                                   # bad argument
                       ("sb_rmsnorm_fwd", (8, 16, 16, None, 1, 8, 8, 8, 1e-5, None)),                 # misaligned
                       ("sb_attention_fwd_pp", (16, 16, None, 70000, 1, 1, 1, 64, 192, 64, 1, 1, 16, None))):   # too large
        rc = calls[name](*args)
        assert rc != 0 and rc == getattr(lib, name)(*args)
        with pytest.raises(_lib.NativeError, match=_lib.ERRORS[rc]):
            _lib.call(name, *args)


def test_wrong_arguments_raise_type_error(calls):
    fn = calls["sb_swiglu_fwd"]
    for args in ((None, None, 0, 0), (None, None, 0, 0, None, None), (None, None, 0.5, 0, None), (None, None, None, 0, None),
                 ("x", None, 0, 0, None)):
        with pytest.raises(TypeError):
            fn(*args)


def test_ctypes_arrays_still_go_through_ctypes():
    lib = _lib.cuda()
    p, handle = ctypes.c_void_p(), (ctypes.c_char * lib.sb_ipc_handle_size())()
    with pytest.raises(_lib.NativeError):                       # no such handle
        _lib.call("sb_ipc_open", handle, ctypes.byref(p))


def test_one_odd_argument_does_not_move_an_entry_point_to_ctypes(calls):
    with pytest.raises(_lib.NativeError):
        _lib.call("sb_swiglu_fwd", None, None, 0, 0, None)
    fast = _lib._calls["sb_swiglu_fwd"]
    assert not isinstance(fast, ctypes._CFuncPtr)
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        _lib.call("sb_swiglu_fwd", None, None, 0.5, 0, None)
    with pytest.raises(_lib.NativeError):
        _lib.call("sb_swiglu_fwd", None, None, np.int32(0), 0, None)
    assert _lib._calls["sb_swiglu_fwd"] is fast


def test_arrays_of_ctypes_are_addresses(calls):
    """The extension takes them as ctypes does; arrays of anything else stay refused."""
    fn, lib = calls["sb_swiglu_fwd"], _lib.cuda()
    arr = (ctypes.c_void_p * 4)(*range(4))
    assert fn(arr, arr, 0, 8, None) == lib.sb_swiglu_fwd(arr, arr, 0, 8, None) != 0        # bad argument: no rows
    for other in (np.zeros(4), bytearray(32), [1, 2]):
        with pytest.raises(TypeError):
            fn(other, None, 0, 0, None)


def test_an_extension_of_another_abi_or_interpreter_is_left_alone(calls, monkeypatch, tmp_path):
    import sysconfig
    assert _build.CALLS_LIB.name == "sb_py_calls" + sysconfig.get_config_var("EXT_SUFFIX")
    with monkeypatch.context() as m:
        m.setattr(_build, "api_digest", lambda: "of a changed api.h")
        assert _lib._native_calls() == {}
    broken = tmp_path / _build.CALLS_LIB.name
    broken.write_bytes(b"not a shared library")
    monkeypatch.setattr(_build, "CALLS_LIB", broken)
    assert _lib._native_calls() == {}                           # and calls go through ctypes
    monkeypatch.setattr(_lib, "_calls", {})
    with pytest.raises(_lib.NativeError):
        _lib.call("sb_swiglu_fwd", None, None, 0, 0, None)


def test_an_extension_that_cannot_be_rebuilt_goes(monkeypatch, tmp_path):
    old = tmp_path / "sb_py_calls.so"
    old.touch()
    monkeypatch.setattr(_build, "CALLS_LIB", old)
    monkeypatch.setattr(_build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})      # no Python.h there
    assert _build.build_calls() is None and not old.exists()


def test_first_use_of_a_missing_library_builds_the_extension_too(monkeypatch, tmp_path):
    built = []
    monkeypatch.setattr(_build, "CUDA_LIB", tmp_path / "missing.so")
    monkeypatch.setattr(_build, "build_cuda", lambda *a, **k: built.append("cuda"))
    monkeypatch.setattr(_build, "build_calls", lambda *a, **k: built.append("calls"))
    monkeypatch.setattr(_lib, "_cuda", None)
    with pytest.raises(_lib.NativeError):                       # the builders here make nothing
        _lib.cuda()
    assert built == ["cuda", "calls"]


@pytest.mark.parametrize("value,on", [(None, True), ("1", True), ("0", False)])
def test_environment_switches_dependent_launches(value, on):
    import os
    import subprocess
    import sys
    env = {k: v for k, v in os.environ.items() if k != "SB_PDL"} | ({"SB_PDL": value} if value else {})
    _lib.cuda()                                                 # is built
    code = (f"import ctypes; f = ctypes.CDLL({str(_build.CUDA_LIB)!r})._ZN2sb18dependent_launchesEv; "
            "f.restype = ctypes.c_bool; print(f())")
    assert subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, check=True).stdout.strip() == str(on)
