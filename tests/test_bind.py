"""The callables of rd_bind.cpp give what ctypes gives (host-side argument errors: no GPU needed)."""
import ctypes as C

import pytest


def test_bound_callables_match_ctypes(rd):
    raw = C.CDLL(rd.LIB_PATH)
    args = {"rd_attn_decode_ws": (16, 32, 48, 64, None, 0, 9, 24, 4, 256, 1 / 16, 7, 1, 1, None, 256, 1 << 20, None),
            "rd_kv_store_rows": (3, 16, 32, 33, 0),
            "rd_attn_prefill_append_fused": (16, 0, 16, 16, 16, 16, None, 16, 4, 0, 4, 24, 4, 256, 1, 64, 10000000, None),
            "rd_attn_merge": (16, 16, -1, 256, 1, None, None)}
    for name, a in args.items():
        ref = getattr(raw, name)
        ref.restype, ref.argtypes = rd.SIGNATURES[name]
        assert getattr(rd.lib, name)(*a) == ref(*a) != rd.OK
        assert getattr(rd.lib, name).__name__ == name
        with pytest.raises((TypeError, C.ArgumentError)):
            getattr(rd.lib, name)(*a[:-1])
        with pytest.raises((TypeError, C.ArgumentError)):
            getattr(rd.lib, name)(object(), *a[1:])
    # what the converter does not take goes to ctypes
    x = C.c_float(1.0)
    assert rd.lib.rd_kv_store_rows(3, C.byref(x), 32, 33, 0) == rd.ERR_SHAPE


def test_module_is_this_interpreters(rd):
    """A module of another interpreter has another name: it is neither loaded nor taken for up to date by make."""
    import os
    import sysconfig
    assert os.path.basename(rd.BIND_PATH) == "_rd_bind" + sysconfig.get_config_var("EXT_SUFFIX")
    if os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h")):
        assert os.path.exists(rd.BIND_PATH) and type(rd.lib.rd_kv_store_rows).__name__ == "builtin_function_or_method"


def recorder(rd, name, calls):
    """A ctypes callback with the signature of an entry: what the bound callable hands over, argument for argument."""
    res, args = rd.SIGNATURES[name]

    def fn(*a):
        calls.append(a)
        return -7
    return C.CFUNCTYPE(res, *args)(fn)


def bound_names(rd):
    return [n for n in rd.SIGNATURES if type(getattr(rd.lib, n)).__name__ == "builtin_function_or_method"]


def install(rd, name, callback):
    import importlib.machinery
    import importlib.util
    loader = importlib.machinery.ExtensionFileLoader("_rd_bind", rd.BIND_PATH)
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_rd_bind", loader))
    loader.exec_module(module)
    return module.install(name, C.cast(callback, C.c_void_p).value, callback)


def test_every_entry_hands_over_every_argument(rd):
    names = bound_names(rd)
    if not names:
        pytest.skip("no Python headers: ctypes serves every call")
    assert len(names) == 26
    for name in names:
        calls = []
        cb = recorder(rd, name, calls)
        fast = install(rd, name, cb)
        types = rd.SIGNATURES[name][1]
        values = [0.5 + i if t is C.c_float else (1 << 40) + 16 * i if t in (C.c_void_p, C.c_size_t, C.c_int64) else 3 + i
                  for i, t in enumerate(types)]
        assert fast(*values) == -7 and list(calls[-1]) == values, name
        # None, 0 and negative numbers; a number for a float; what ctypes does with numbers out of range
        other = [None if t is C.c_void_p else 7 if t is C.c_float else -5 if t in (C.c_int, C.c_int64) else 0 for t in types]
        assert fast(*other) == -7 and list(calls[-1]) == other, name
        wide = [(1 << 35) + 9 if t is C.c_int else v for t, v in zip(types, values)]
        assert fast(*wide) == cb(*wide) == -7 and calls[-2] == calls[-1], name
        with pytest.raises(TypeError):
            fast(*values[:-1])
        with pytest.raises((TypeError, C.ArgumentError)):
            fast(object(), *values[1:])


def test_callables_of_two_libraries_stay_apart(rd):
    if not bound_names(rd):
        pytest.skip("no Python headers: ctypes serves every call")
    first, second = [], []
    a, b = recorder(rd, "rd_kv_store_rows", first), recorder(rd, "rd_kv_store_rows", second)
    fa, fb = install(rd, "rd_kv_store_rows", a), install(rd, "rd_kv_store_rows", b)
    assert fa(1, 16, 32, 64, 0) == -7 and (len(first), len(second)) == (1, 0)
    assert fb(1, 16, 32, 64, 0) == -7 and (len(first), len(second)) == (1, 1)
    assert rd.lib.rd_kv_store_rows(3, 16, 32, 33, 0) == rd.ERR_SHAPE     # the product's own is what it was
