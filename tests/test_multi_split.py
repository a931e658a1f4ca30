"""The key split of a many-sequence call (host arithmetic, no GPU): what a plan's items write fits the workspace."""
import ctypes as C
import random

import pytest

SMS = 148


def splits(rd, t, q_len, nkv, kt, vt):
    n = len(t)
    out = (C.c_int32 * n)()
    rd.check(rd.lib.rd_attn_multi_split((C.c_int32 * n)(*t), n, q_len, nkv, kt, vt, SMS, out))
    return list(out)


@pytest.mark.parametrize("nkv", [1, 2, 4])
@pytest.mark.parametrize("q_len", [1, 2, 3, 4, 5, 6, 7, 8, 9, 13, 16, 17, 40])
def test_records_and_items_fit(rd, nkv, q_len):
    rng = random.Random(q_len)
    shapes = [[9000], [200000], [q_len - 1], [131071] * 2] + [
        [rng.randint(q_len - 1, most) for _ in range(n)] for n in (1, 3, 17, 64, 200, 700) for most in (q_len + 50, 4000, 60000)]
    for t in shapes:
        for kt, vt in ((3, 3), (2, 1), (0, 0)):
            s = splits(rd, t, q_len, nkv, kt, vt)
            room = 4 * SMS + len(t) * q_len      # records per head, and items: rd_attn_multi_workspace_bytes
            tile = 64 if q_len > 1 else 16
            chunks = (q_len + 7) // 8
            assert all(1 <= x <= max(1, (last + tile) // tile) for x, last in zip(s, t))
            assert sum(s) * q_len <= room and sum(s) * chunks <= room, (len(t), max(t), kt, vt)


def test_split_arguments(rd):
    L, t, out = rd.lib, (C.c_int32 * 1)(99), (C.c_int32 * 1)()
    assert L.rd_attn_multi_split(t, 1, 1, 4, 3, 9, SMS, out) == rd.ERR_TYPE
    assert L.rd_attn_multi_split(t, 1, 1, 3, 3, 3, SMS, out) == rd.ERR_UNSUPPORTED
    assert L.rd_attn_multi_split(t, 0, 1, 4, 3, 3, SMS, out) == rd.ERR_SHAPE
    assert L.rd_attn_multi_split(t, 1, 101, 4, 3, 3, SMS, out) == rd.ERR_SHAPE
    assert L.rd_attn_multi_split(None, 1, 1, 4, 3, 3, SMS, out) == rd.ERR_NULL
    assert L.rd_attn_multi_split(t, 1, 1, 4, 3, 3, SMS, None) == rd.ERR_NULL
