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
