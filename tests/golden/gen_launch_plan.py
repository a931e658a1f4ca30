"""Writes b200_launch_plan.txt: which launch the library takes for decode calls and blocks of tokens at and around the
lengths where it changes, and the key split of many sequences, on 148 SMs. Needs only the built library (host
arithmetic, no GPU):

    python tests/golden/gen_launch_plan.py            # rewrite the golden file
    python tests/golden/gen_launch_plan.py --print    # print the table instead
"""
import ctypes as C
import importlib
import os
import random
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(os.path.dirname(HERE)))
NAMES = ("f32", "f16", "q8_0", "q4_0", "q5_0", "q4_1")
FORMS = ("clusters", "heads", "all", "block")
KEYS = (0, 1, 256, 257, 895, 897, 1408, 1409, 1793, 2817, 3584, 3585, 5632, 5633, 24576, 24577, 131001, -1)


def table():
    rd = importlib.import_module("rdna4-infer_b200")
    L = rd.lib
    form, splits, ctas = C.c_int(), C.c_int(), C.c_int()

    def plan(n_keys, n_tok, nkv, kt, vt):
        rd.check(L.rd_attn_launch_plan(n_keys, n_tok, nkv, kt, vt, 148, C.addressof(form), C.addressof(splits),
                                       C.addressof(ctas)))
        return f"{FORMS[form.value]}:{splits.value}:{ctas.value}"

    lines = ["# form:splits:CTAs of a decode launch; K V kv_heads | keys " + " ".join(map(str, KEYS))]
    for nkv in (4, 2, 1):
        for kt in range(6):
            for vt in range(6):
                lines.append(f"{NAMES[kt]} {NAMES[vt]} {nkv} | " + " ".join(plan(n, 1, nkv, kt, vt) for n in KEYS))
    lines.append("# blocks of 2 .. 9, 16, 17, 40 tokens; kv_heads |")
    for nkv in (4, 2, 1):
        lines.append(f"{nkv} | " + " ".join(plan(-1, t, nkv, 3, 3) for t in (2, 3, 4, 5, 6, 7, 8, 9, 16, 17, 40)))
    lines.append("# many sequences: count shortest longest tokens kv_heads K V | splits by length (last key: splits)")
    for n, lo, hi, q_len, nkv, kt, vt in ((1, 9000, 9000, 1, 4, 3, 3), (2, 5000, 6000, 1, 4, 3, 2), (8, 4000, 30000, 1, 4, 2, 1),
                                          (64, 1024, 32768, 1, 4, 2, 1), (64, 1024, 32768, 4, 4, 2, 1), (5, 10, 900, 5, 4, 3, 2),
                                          (40, 9, 80, 9, 4, 3, 2), (3, 2000, 9000, 8, 1, 1, 1), (1, 14000, 14000, 5, 1, 3, 2)):
        rng = random.Random(n)
        t = sorted(rng.randint(lo, hi) - 1 for _ in range(n))
        out = (C.c_int32 * n)()
        rd.check(L.rd_attn_multi_split((C.c_int32 * n)(*t), n, q_len, nkv, kt, vt, 148, out))
        shown = sorted({0, n // 3, 2 * n // 3, n - 1})
        lines.append(f"{n} {lo} {hi} {q_len} {nkv} {NAMES[kt]} {NAMES[vt]} | {sum(out)} "
                     + " ".join(f"{t[i]}:{out[i]}" for i in shown))
    return "\n".join(lines) + "\n"


if __name__ == "__main__":
    if "--print" in sys.argv:
        sys.stdout.write(table())
    else:
        with open(os.path.join(HERE, "b200_launch_plan.txt"), "w") as f:
            f.write(table())
