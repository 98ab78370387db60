"""The generated call module gives what ctypes gives, and leaves to ctypes what it does not convert."""
import ctypes

import pytest

from flashrt_b200 import _lib


def test_native_calls_agree_with_ctypes():
    lib = _lib.load()
    native = pytest.importorskip("flashrt_b200._native_calls")
    assert all(hasattr(native, n) for n in _lib.exported_names())
    args = [0, None, None, 0, None, None, 0, 0, None, 10, 100, 1e-6, 0, 0, 0]        # NULL residual: refused on the host
    assert native.frt_b200_norm_fp8(*args) == lib.frt_b200_norm_fp8(*args) == -1
    args[11] = 1                                                                     # an int where a float is declared
    assert native.frt_b200_norm_fp8(*args) == -1
    for i, bad in ((0, ctypes.c_void_p(0)), (0, -1), (9, 1.5), (11, None)):
        assert native.frt_b200_norm_fp8(*args[:i], bad, *args[i + 1:]) is NotImplemented
    assert native.frt_b200_norm_fp8(*args[:-1]) is NotImplemented
    assert _lib.call_status("frt_b200_norm_fp8", ctypes.c_void_p(0), *args[1:]) == -1
    with pytest.raises(ctypes.ArgumentError):
        _lib.call_status("frt_b200_norm_fp8", *args[:9], 1.5, *args[10:])
    with pytest.raises(_lib.KernelError):
        _lib.call("frt_b200_norm_fp8", *args)


def test_call_module_belongs_to_one_interpreter(monkeypatch, tmp_path):
    """The module's file carries the interpreter's tag, and where it cannot be built again neither a stale one nor one that any
    interpreter would import stays behind."""
    import os
    import sysconfig
    from flashrt_b200 import _build
    native = pytest.importorskip("flashrt_b200._native_calls")
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    assert suffix != ".so" and native.__file__ == _build.CALLS and _build.CALLS.endswith("_native_calls" + suffix)
    calls, untagged = tmp_path / ("_native_calls" + suffix), tmp_path / "_native_calls.so"
    monkeypatch.setattr(_build, "CALLS", str(calls))
    monkeypatch.setattr(_build.shutil, "which", lambda name: None)
    for f in (calls, untagged):
        f.write_bytes(b"")
        os.utime(f, (1, 1))
    assert _build.build_calls() is None and not calls.exists() and not untagged.exists()
