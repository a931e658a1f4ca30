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
