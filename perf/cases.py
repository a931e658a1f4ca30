"""The work that a user of this library has it do, as a list of cases.

One pass is what an engine runs between two samplings: the attention of one decode step, one
verify block or one prefill chunk, through the full-attention layers of the model (24 query and
4 KV heads, head_dim 256, 64 rotated dims, sigmoid output gate), every layer with a cache of its
own, or one batched step over many sequences. All calls go through the C ABI of
include/rd_attn.h, one after another on the current stream, as an engine's layer loop makes them.

Kinds:
  step     one new token: rd_pre_attn_fused (split, norm, RoPE, cache append), rd_attn_decode_ws
  append   one new token whose rows are ready: rd_attn_decode_append_ws
  verify   a block of drafted tokens: rd_pre_attn_fused, rd_attn_split_batch, rd_sigmoid_gate
  prefill  a prompt chunk over f16 caches: rd_attn_prefill_append_fused
  typed    a prompt chunk over quantized caches: rd_kv_append, rd_attn_prefill_typed
  multi    many sequences in one call: rd_attn_decode_multi (q_len 1 decodes, above 1 verifies)
"""
import ctypes
import importlib
import math
import random

import torch

rd = importlib.import_module("rdna4-infer_b200")

NH, NKV, HD = 24, 4, 256
N_ROT, FREQ_BASE, EPS, SCALE = 64, 1e7, 1e-6, 1.0 / 16.0
LAYERS = 16                       # full-attention layers of the model
TYPES = {"f32": rd.F32, "f16": rd.F16, "q8_0": rd.Q8_0, "q4_0": rd.Q4_0, "q5_0": rd.Q5_0, "q4_1": rd.Q4_1}
# K / V type pairs that engines serve with, and the share of the drawn cases that each has
PAIRS = (("f16", "f16", 3), ("q8_0", "q8_0", 3), ("q4_0", "q4_0", 3), ("q5_0", "q4_1", 2), ("q8_0", "f16", 1),
         ("q8_0", "q4_0", 1))
MOST_BYTES = 3.6e9                # cache bytes that a drawn pass may walk
MOST_FLOPS = 1.5e12               # and what a drawn prefill pass may compute


def listed():
    return [
        # the first tokens of a chat: everything is launches, latency and host work
        dict(name="step f16 137 keys", kind="step", k="f16", v="f16", keys=137, layers=LAYERS),
        # an ordinary chat turn on plain f16 caches
        dict(name="step f16 4096 keys", kind="step", k="f16", v="f16", keys=4096, layers=LAYERS),
        # a long conversation on 8-bit caches
        dict(name="step q8_0 32768 keys", kind="step", k="q8_0", v="q8_0", keys=32768, layers=LAYERS),
        # the default pair of long-context serving, at an odd length
        dict(name="step q5_0/q4_1 65537 keys", kind="step", k="q5_0", v="q4_1", keys=65537, layers=LAYERS),
        # the longest context: one token at position 131000 on 4-bit caches
        dict(name="append q4_0 131001 keys", kind="append", k="q4_0", v="q4_0", keys=131001, layers=LAYERS),
        # speculative decoding: four drafted tokens and the last accepted one are checked at once
        dict(name="verify 5 q4_0 20011 keys", kind="verify", k="q4_0", v="q4_0", keys=20011, q_len=5, layers=LAYERS),
        # a fresh prompt's only chunk
        dict(name="prefill 512 at 0", kind="prefill", k="f16", v="f16", n_q=512, pos0=0, layers=LAYERS),
        # a late chunk of a long prompt
        dict(name="prefill 512 at 7680", kind="prefill", k="f16", v="f16", n_q=512, pos0=7680, layers=LAYERS),
        # the ragged last chunk of a prompt over quantized caches
        dict(name="typed q8_0 389 at 11957", kind="typed", k="q8_0", v="q8_0", n_q=389, pos0=11957, layers=LAYERS),
        # a whole long prompt at once
        dict(name="prefill 8192 at 0", kind="prefill", k="f16", v="f16", n_q=8192, pos0=0, layers=1),
        # a server's batch of 64 conversations of all lengths: one decode step of one layer
        dict(name="multi 64 q8_0/f16", kind="multi", k="q8_0", v="f16", n_seq=64, q_len=1, shortest=1024,
             longest=32768, len_seed=7, layers=1),
        # the same batch verifying blocks of four tokens
        dict(name="multi 64 q8_0/f16 verify 4", kind="multi", k="q8_0", v="f16", n_seq=64, q_len=4, shortest=1024,
             longest=32768, len_seed=7, layers=1),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _pair(rng, quantized=False):
    pairs = [p for p in PAIRS if not quantized or p[:2] != ("f16", "f16")]
    k, v, _ = rng.choices(pairs, weights=[p[2] for p in pairs])[0]
    return k, v


def _key_bytes(case):
    return NKV * (rd.row_bytes(TYPES[case["k"]]) + rd.row_bytes(TYPES[case["v"]]))


def draw(rng):
    kind = rng.choices(("step", "append", "verify", "prefill", "typed", "multi"), weights=(5, 2, 2, 3, 2, 3))[0]
    if kind in ("step", "append", "verify"):
        k, v = _pair(rng)
        c = dict(kind=kind, k=k, v=v, layers=LAYERS)
        c["keys"] = _log_int(rng, 64, min(131072, int(MOST_BYTES / LAYERS / _key_bytes(c))))
        if kind == "verify":
            c["q_len"] = rng.randint(2, 8)
            c["keys"] = min(c["keys"], 65536)
        return c
    if kind in ("prefill", "typed"):
        k, v = _pair(rng, True) if kind == "typed" else ("f16", "f16")
        c = dict(kind=kind, k=k, v=v, n_q=_log_int(rng, 24, 8192 if kind == "prefill" else 1024), layers=LAYERS)
        c["pos0"] = 0 if rng.random() < 0.3 else _log_int(rng, 64, 24576)
        while _flops(dict(c, layers=1)) > MOST_FLOPS:    # a long chunk after a long prefix: start earlier
            c["pos0"] = c["pos0"] * 2 // 3
        c["layers"] = max(1, min(LAYERS, int(MOST_FLOPS / _flops(dict(c, layers=1)))))
        return c
    k, v = _pair(rng)
    c = dict(kind="multi", k=k, v=v, n_seq=_log_int(rng, 2, 128), q_len=rng.choice((1, 1, 1, 2, 3, 4, 5)),
             shortest=_log_int(rng, 64, 2048), len_seed=rng.randint(0, 1 << 20), layers=1)
    c["longest"] = c["shortest"] + _log_int(rng, 64, 32768)
    room = MOST_BYTES / _key_bytes(c) / c["n_seq"]
    c["longest"] = max(c["shortest"] + 1, min(c["longest"], int(room)))
    return c


def _lengths(case):
    r = random.Random(case["len_seed"])
    return [r.randint(case["shortest"], case["longest"]) for _ in range(case["n_seq"])]


# ---- inputs ---------------------------------------------------------------------------------
class _Rand:
    """N(0, 1) device tensors from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def __call__(self, *shape):
        return torch.randn(*shape, device="cuda", generator=self.g)


def _filled_caches(rand, kv_type, n, rows):
    """[n][rows][bytes of a key]: N(0, 1) rows through the library's own quantizer."""
    row = NKV * rd.row_bytes(kv_type)
    cache = torch.empty(n, rows, row, dtype=torch.uint8, device="cuda")
    flat = cache.view(n * rows, row)
    st, step = rd.stream_ptr(), 1 << 15
    for r0 in range(0, n * rows, step):
        m = min(step, n * rows - r0)
        rd.check(rd.lib.rd_kv_store_rows(kv_type, rd.ptr(rand(m, NKV * HD)), rd.ptr(flat[r0]), m * NKV * HD, st))
    return cache


def prepare(case, seed):
    return {"step": _prepare_step, "verify": _prepare_step, "append": _prepare_append, "prefill": _prepare_prefill,
            "typed": _prepare_prefill, "multi": _prepare_multi}[case["kind"]](case, _Rand(seed))


# A state holds the calls of a pass (function, arguments up to the stream), what they return into,
# and the tensors behind the pointers.
def _state(calls, outputs, *keep):
    return {"calls": calls, "outputs": outputs, "keep": keep}


def _prepare_step(case, rand):
    L, kt, vt, n, keys = rd.lib, TYPES[case["k"]], TYPES[case["v"]], case["layers"], case["keys"]
    q_len = case.get("q_len", 1)
    row0 = keys - q_len
    kc, vc = _filled_caches(rand, kt, n, keys), _filled_caches(rand, vt, n, keys)
    qg, ks, vs = rand(n, q_len, NH, 2 * HD), rand(n, q_len, NKV, HD), rand(n, q_len, NKV, HD)
    qw, kw = 1 + 0.1 * rand(n, HD), 1 + 0.1 * rand(n, HD)
    q, gate, out = (torch.empty(n, q_len, NH, HD, device="cuda") for _ in range(3))
    pos = torch.arange(row0, keys, dtype=torch.int32, device="cuda")
    nb = L.rd_attn_workspace_bytes(1, NH, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    splits = L.rd_attn_splits_for(keys, kt, vt, NH, 0)
    calls, p = [], rd.ptr
    for i in range(n):
        calls.append((L.rd_pre_attn_fused, (p(qg[i]), p(ks[i]), p(vs[i]), p(qw[i]), p(kw[i]), EPS, p(q[i]), p(gate[i]),
                                            p(kc[i, row0]), p(vc[i, row0]), kt, vt, p(pos), q_len, NH, NKV, HD, N_ROT,
                                            FREQ_BASE)))
        if case["kind"] == "step":
            calls.append((L.rd_attn_decode_ws, (p(q[i]), p(kc[i]), p(vc[i]), p(out[i]), None, 0, keys - 1, NH, NKV, HD,
                                                SCALE, kt, vt, splits, p(gate[i]), p(ws), nb)))
        else:
            calls.append((L.rd_attn_split_batch, (p(q[i]), p(kc[i]), p(vc[i]), p(out[i]), None, p(pos), q_len, NH, NKV,
                                                  HD, SCALE, kt, vt, splits)))
            calls.append((L.rd_sigmoid_gate, (p(gate[i]), p(out[i]), q_len * NH * HD)))
    return _state(calls, {"out": out, "gate": gate, "q": q, "k_rows": kc[:, row0:], "v_rows": vc[:, row0:]},
                  qg, ks, vs, qw, kw, pos, ws, kc, vc)


def _prepare_append(case, rand):
    L, kt, vt, n, keys = rd.lib, TYPES[case["k"]], TYPES[case["v"]], case["layers"], case["keys"]
    kc, vc = _filled_caches(rand, kt, n, keys), _filled_caches(rand, vt, n, keys)
    q, gate, ks, vs = rand(n, NH, HD), rand(n, NH, HD), rand(n, NKV, HD), rand(n, NKV, HD)
    out = torch.empty(n, NH, HD, device="cuda")
    nb = L.rd_attn_workspace_bytes(1, NH, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    p = rd.ptr
    calls = [(L.rd_attn_decode_append_ws, (p(q[i]), p(ks[i]), p(vs[i]), p(kc[i]), p(vc[i]), p(out[i]), keys - 1, NH,
                                           NKV, HD, SCALE, kt, vt, p(gate[i]), p(ws), nb)) for i in range(n)]
    return _state(calls, {"out": out, "gate": gate, "k_rows": kc[:, keys - 1], "v_rows": vc[:, keys - 1]},
                  q, ks, vs, ws, kc, vc)


def _prepare_prefill(case, rand):
    L, kt, vt, n, n_q, row0 = rd.lib, TYPES[case["k"]], TYPES[case["v"]], case["layers"], case["n_q"], case["pos0"]
    keys = row0 + n_q
    kc, vc = _filled_caches(rand, kt, n, keys), _filled_caches(rand, vt, n, keys)
    q, gate, ks, vs = rand(n, n_q, NH, HD), rand(n, n_q, NH, HD), rand(n, n_q, NKV, HD), rand(n, n_q, NKV, HD)
    out = torch.empty(n, n_q, NH, HD, device="cuda")
    pos = torch.arange(row0, keys, dtype=torch.int32, device="cuda")
    calls, p, ws = [], rd.ptr, None
    if case["kind"] == "typed":
        nb = L.rd_attn_prefill_workspace_bytes(kt, vt, n_q, keys, NH, NKV, HD)
        ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    for i in range(n):
        if ws is None:
            calls.append((L.rd_attn_prefill_append_fused, (p(q[i]), p(ks[i]), p(vs[i]), p(kc[i]), p(vc[i]), p(out[i]),
                                                           p(gate[i]), p(pos), n_q, row0, keys, NH, NKV, HD, SCALE,
                                                           N_ROT, FREQ_BASE)))
        else:
            calls.append((L.rd_kv_append, (kt, vt, p(ks[i]), p(vs[i]), p(kc[i, row0]), p(vc[i, row0]), n_q, NKV, HD,
                                           p(pos), N_ROT, FREQ_BASE)))
            calls.append((L.rd_attn_prefill_typed, (p(q[i]), p(kc[i]), p(vc[i]), p(out[i]), p(gate[i]), p(pos), n_q,
                                                    keys, NH, NKV, HD, SCALE, kt, vt, N_ROT, FREQ_BASE, p(ws), nb)))
    return _state(calls, {"out": out, "k_rows": kc[:, row0:], "v_rows": vc[:, row0:]}, q, gate, ks, vs, pos, ws, kc, vc)


def _prepare_multi(case, rand):
    L, kt, vt, q_len = rd.lib, TYPES[case["k"]], TYPES[case["v"]], case["q_len"]
    lens = _lengths(case)
    n = len(lens)
    q, gate = rand(n, q_len, NH, HD), rand(n, q_len, NH, HD)
    out = torch.empty(n, q_len, NH, HD, device="cuda")
    kcs = [_filled_caches(rand, kt, 1, m) for m in lens]
    vcs = [_filled_caches(rand, vt, 1, m) for m in lens]
    seqs = (rd.AttnSeq * n)()
    for i, m in enumerate(lens):
        seqs[i].q, seqs[i].k, seqs[i].v = rd.ptr(q[i]), rd.ptr(kcs[i]), rd.ptr(vcs[i])
        seqs[i].out, seqs[i].gate, seqs[i].t = rd.ptr(out[i]), rd.ptr(gate[i]), m - 1
    nb = L.rd_attn_multi_workspace_bytes(n, q_len, NH, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    calls = [(L.rd_attn_decode_multi, (ctypes.addressof(seqs), n, q_len, NH, NKV, HD, SCALE, kt, vt, rd.ptr(ws), nb))]
    return _state(calls, {"out": out, "gate": gate}, q, seqs, ws, kcs, vcs)


def run(state):
    st = torch.cuda.current_stream().cuda_stream
    for fn, args in state["calls"]:
        rc = fn(*args, st)
        if rc != rd.OK:
            rd.check(rc, fn.__name__)
    return state["outputs"]


# ---- what a pass cannot do without -------------------------------------------------------------
def _attended(case):
    """(keys read, query-key pairs) of one layer."""
    if case["kind"] == "multi":
        lens, b = _lengths(case), case["q_len"]
        return sum(lens), sum(b * m - b * (b - 1) // 2 for m in lens)
    if case["kind"] in ("prefill", "typed"):
        n_q, pos0 = case["n_q"], case["pos0"]
        return pos0 + n_q, n_q * pos0 + n_q * (n_q + 1) // 2
    b = case.get("q_len", 1)
    return case["keys"], b * case["keys"] - b * (b - 1) // 2


def _flops(case):
    return 4.0 * HD * NH * _attended(case)[1] * case["layers"]


def work(case):
    keys, _ = _attended(case)
    head, kv = NH * HD * 4, 2 * NKV * HD * 4            # bytes of a token's heads and of its new K and V rows
    tokens = {"multi": case.get("n_seq", 1) * case.get("q_len", 1), "prefill": case.get("n_q"),
              "typed": case.get("n_q")}.get(case["kind"], case.get("q_len", 1))
    per_token = {"step": 5 * head + kv, "verify": 5 * head + kv,   # q and gate in; q, gate and out written
                 "append": 4 * head + kv,                          # q and gate in; gate and out written
                 "prefill": 3 * head + kv, "typed": 3 * head + kv,  # q and gate in; out written
                 "multi": 4 * head}[case["kind"]]
    if case["kind"] != "multi":
        per_token += _key_bytes(case)                    # the new rows are stored too
    return {"bytes": float(case["layers"] * (keys * _key_bytes(case) + tokens * per_token)), "flops": _flops(case)}


def tolerance(case):
    # The contractions take f16 operands (weights, and the values of the caches) with f32 sums:
    # 2^-11 for each operand. Stored rows are the quantizers' bytes and stay the same.
    return {"rel": 2e-3, "max": 5e-2}
