"""The typed callers behind ``ops._lib.call`` (host only: no kernel is launched)."""
import ctypes

import pytest

from prometheus_b200.ops import _lib

pytestmark = pytest.mark.skipif(not (_lib.available() and _lib._CALL_PATH.exists()), reason="libraries not built")


def test_plain_symbols_get_a_typed_caller_and_host_array_ones_do_not():
    lib = _lib.load()
    for name in _lib._SIGS:
        if hasattr(lib, name):
            assert (_lib._bind(name) is not getattr(lib, name)) == (name in _lib._PLAIN), name
    assert "pb_cp_push" not in _lib._PLAIN and "pb_gemm_bf16_ag" not in _lib._PLAIN
    _lib._bound.clear()


@pytest.mark.parametrize("args", [(1, 128), (300, 2048), (1 << 20, 4096), (True, 8)])
def test_values_agree_with_the_foreign_call(args):
    fn = _lib._bind("pb_rmsnorm_bwd_nparts")
    assert fn(*args) == _lib.query("pb_rmsnorm_bwd_nparts", *args)
    assert _lib._bind("pb_sumsq_nparts")(args[0] << 20) == _lib.query("pb_sumsq_nparts", args[0] << 20)


def test_argument_checks_and_status_codes():
    fn = _lib._bind("pb_sigmoid")
    with pytest.raises(TypeError):
        fn(1, 2)
    for bad in (("x", None, 1, 0), (1.5, None, 1, 0), (None, None, "n", 0), (ctypes.c_void_p(1), None, 1, 0)):
        with pytest.raises(TypeError):
            fn(*bad)
    with pytest.raises(RuntimeError, match="pb_scale_cast failed"):      # refused by the host check
        _lib.call("pb_scale_cast", None, None, None, 0, None)


def test_call_takes_and_refuses_what_the_foreign_call_does():
    """A symbol with host checks only on this path (n = 0 is refused before a pointer is looked at)."""
    numpy = pytest.importorskip("numpy")
    n0 = "pb_scale_cast failed with code"
    for args in ((ctypes.c_void_p(16), None, None, 0, None), (None, ctypes.byref(ctypes.c_int(3)), None, 0, None),
                 (None, None, None, ctypes.c_long(0), None), (None, None, None, 1 << 64, None), (16, 16, 16, False, 0),
                 (None, None, None, numpy.int64(0), None)):
        with pytest.raises(RuntimeError, match=n0):
            _lib.call("pb_scale_cast", *args)
    for args in ((1.5, None, None, 0, None), (None, None, None, "0", None), (None, None, None, 0.0, None)):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            _lib.call("pb_scale_cast", *args)
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            getattr(_lib.load(), "pb_scale_cast")(*args)


@pytest.mark.parametrize("stale", [False, True])
def test_a_missing_or_stale_caller_module_is_reported_once(stale, monkeypatch, tmp_path):
    """Launches still work, at twice the host time: that must not go unnoticed."""
    import types
    import warnings

    monkeypatch.setattr(_lib, "_bound", {})
    monkeypatch.setattr(_lib, "_warned", False, raising=False)
    monkeypatch.setattr(_lib, "_CALL_PATH", tmp_path / "absent.so")
    monkeypatch.setattr(_lib, "_binder", types.SimpleNamespace(bind=lambda address, sig: None) if stale else None)
    with pytest.warns(RuntimeWarning, match="missing or older"):
        fn = _lib._bind("pb_rmsnorm_bwd_nparts")
    assert fn(300, 2048) == _lib.query("pb_rmsnorm_bwd_nparts", 300, 2048)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        _lib._bind("pb_sigmoid")
