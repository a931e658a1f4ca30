"""Which launch a call takes, and how many sequences are split, against the committed table (host arithmetic, no GPU)."""
import ctypes as C
import os

from tests.golden.gen_launch_plan import table

HERE = os.path.dirname(os.path.abspath(__file__))


def test_launches_match_committed_table():
    assert table() == open(os.path.join(HERE, "golden", "b200_launch_plan.txt")).read()


def test_launch_plan_arguments(rd):
    f = rd.lib.rd_attn_launch_plan
    form, splits, ctas = C.c_int(), C.c_int(), C.c_int()
    out = (C.addressof(form), C.addressof(splits), C.addressof(ctas))
    assert f(131001, 1, 4, 3, 3, 148, *out) == rd.OK and (form.value, splits.value, ctas.value) == (2, 148, 148)
    assert f(137, 1, 4, 1, 1, 148, *out) == rd.OK and (form.value, splits.value, ctas.value) == (0, 8, 32)
    assert f(20011, 5, 4, 3, 3, 148, *out) == rd.OK and (form.value, splits.value, ctas.value) == (3, 37, 148)
    assert f(8192, 1, 4, 2, 2, 148, None, None, None) == rd.OK
    assert f(10, 1, 4, 6, 3, 148, *out) == rd.ERR_TYPE and f(10, 0, 4, 3, 3, 148, *out) == rd.ERR_SHAPE
    assert f(10, 1, 3, 3, 3, 148, *out) == rd.ERR_UNSUPPORTED


def test_prefill_launch_plan(rd):
    """rd_attn_prefill_launch_plan: (tile heads, tile tokens, key splits, CTAs) on 148 SMs; argument errors."""
    a = [C.c_int() for _ in range(4)]
    f = rd.lib.rd_attn_prefill_launch_plan
    plan = lambda n_q, keys, nh=24, sms=148: (f(n_q, keys, nh, sms, *[C.addressof(x) for x in a]), *[x.value for x in a])
    assert plan(1, 1) == (0, 1, 128, 1, 24) and plan(512, 512) == (0, 1, 128, 1, 96)   # whole tiles, no records
    assert plan(24, 24024) == (0, 3, 42, 18, 144) and plan(130, 4130) == (0, 3, 42, 4, 128)
    assert plan(512, 4096) == (0, 1, 128, 1, 96) and plan(8192, 8192) == (0, 1, 128, 1, 1536)
    assert plan(389, 12346) == (0, 3, 42, 0, 224) and plan(512, 8192) == (0, 1, 128, 0, 242)   # balanced: parts
    assert f(0, 1, 24, 148, *[None] * 4) == rd.ERR_SHAPE and f(1, 0, 24, 148, *[None] * 4) == rd.ERR_SHAPE
    assert f(1, 1, 5, 148, *[None] * 4) == rd.ERR_UNSUPPORTED and f(1, 1, 6, 148, *[None] * 4) == rd.OK
