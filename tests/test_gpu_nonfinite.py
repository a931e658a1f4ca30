"""Values that are not finite reach the outputs that they belong to, and no others; against the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.conftest import check_attn

pytestmark = pytest.mark.gpu
NKV, NH, HD = 4, 24, 256
F16, Q4_1 = 1, 5
ROW = {F16: 512, Q4_1: 160}


@pytest.fixture(scope="module")
def G(cuda):
    from tests import gpu_util
    return gpu_util


def make(oracle, seed, n, kt, vt, n_tok):
    rng = np.random.default_rng(seed)
    K, V = (rng.standard_normal((n, NKV, HD)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((n_tok, NH, HD)).astype(np.float32)
    return q, oracle.kv_store_rows(kt, K), oracle.kv_store_rows(vt, V)


def plant(vc, want, vt, row, kvh, pos):
    """+inf as dim 37 of a V row (f16), or as the minimum of its second block (q4_1: 32 dims); and in what the
    tokens that attend the row give. (The oracle itself widens the bytes of infinity to 65536, as the reference does.)"""
    at, dims = (2 * 37, slice(37, 38)) if vt == F16 else (20 + 2, slice(32, 64))
    vc.reshape(-1, NKV, ROW[vt])[row, kvh, at:at + 2] = (0x00, 0x7C)
    want[np.asarray(pos) >= row, 6 * kvh:6 * kvh + 6, dims] = np.inf


def same(got, want, what):
    fin = np.isfinite(want)
    assert not fin.all() and (np.isfinite(got) == fin).all(), what
    assert np.array_equal(got[~fin], want[~fin], equal_nan=True), what
    check_attn(np.where(fin, got, 0), np.where(fin, want, 0), what=what)


@pytest.mark.parametrize("kt,vt", [(F16, F16), (2, F16), (Q4_1, Q4_1)])
@pytest.mark.parametrize("n,n_tok", [(5, 5), (70, 3), (400, 2), (400, 8), (9000, 5), (300, 11)])
def test_block_tokens_do_not_see_later_rows(G, oracle, kt, vt, n, n_tok):
    q, kc, vc = make(oracle, n + n_tok, n, kt, vt, n_tok)
    pos = np.arange(n - n_tok, n, dtype=np.int32)
    want = oracle.attn(q, kc, vc, pos, NKV, 1 / 16, kt, vt)
    plant(vc, want, vt, n - 1, 2, pos)
    plant(vc, want, vt, n - 2, 0, pos)
    same(G.attn_batch(q, kc, vc, pos, kt, vt, n_splits=4), want, f"{n_tok} tokens, {n} keys")
    G.status_ok()


def test_block_ragged_positions_and_inner_rows(G, oracle):
    n, kt, vt = 500, 2, F16
    q, kc, vc = make(oracle, 1, n, kt, vt, 7)
    pos = np.array([499, 0, 64, 130, 129, 131, 320], dtype=np.int32)
    want = oracle.attn(q, kc, vc, pos, NKV, 1 / 16, kt, vt)
    for row, kvh in ((130, 1), (131, 2), (499, 3), (65, 0)):
        plant(vc, want, vt, row, kvh, pos)
    same(G.attn_batch(q, kc, vc, pos, kt, vt), want, "ragged")


def test_block_of_many_sequences(G, oracle):
    rd, lib = G.rd, G.lib
    q_len, kt, vt, lens = 4, 2, F16, (4, 37, 900)
    seqs, keep = (rd.AttnSeq * len(lens))(), []
    for i, n in enumerate(lens):
        q, kc, vc = make(oracle, n, n, kt, vt, q_len)
        pos = np.arange(n - q_len, n, dtype=np.int32)
        want = oracle.attn(q, kc, vc, pos, NKV, 1 / 16, kt, vt)
        plant(vc, want, vt, n - 1, i, pos)
        d = [G.dev(q), G.dev(kc), G.dev(vc), G.poison(q.shape)]
        seqs[i].q, seqs[i].k, seqs[i].v, seqs[i].out = (rd.ptr(x) for x in d)
        seqs[i].t = n - 1
        keep.append((d, want, n))
    nb = lib.rd_attn_multi_workspace_bytes(len(lens), q_len, NH, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    rd.check(lib.rd_attn_decode_multi(C.addressof(seqs), len(lens), q_len, NH, NKV, HD, 1 / 16, kt, vt, rd.ptr(ws), nb, G.st()))
    torch.cuda.synchronize()
    for d, want, n in keep:
        same(G.host(d[3]), want, f"{n} keys")


@pytest.mark.parametrize("append", [False, True])
@pytest.mark.parametrize("kt,vt", [(F16, F16), (2, F16), (Q4_1, Q4_1)])
@pytest.mark.parametrize("n", [1, 2, 17, 137, 255, 4100, 6000])
def test_infinite_last_row_of_a_step(G, oracle, kt, vt, n, append):
    """The slot of the last key has rows behind it, with weight 0: they must not turn an infinite last row into NaN."""
    rd, lib = G.rd, G.lib
    q, kc, vc = make(oracle, n, n, kt, vt, 1)
    want = oracle.attn(q, kc, vc, [n - 1], NKV, 1 / 16, kt, vt)
    dq, out = G.dev(q), G.poison(q.shape)
    nb = lib.rd_attn_workspace_bytes(1, NH, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    if append:   # f32 values that a new f16 row saturates; q4_1 blocks of one value have it as their minimum
        kn, vn = (np.random.default_rng(n).standard_normal((NKV, HD)).astype(np.float32) for _ in range(2))
        kc.reshape(n, -1)[n - 1] = oracle.kv_store_rows(kt, kn).reshape(-1)
        vc.reshape(n, -1)[n - 1] = oracle.kv_store_rows(vt, vn).reshape(-1)
        want = oracle.attn(q, kc, vc, [n - 1], NKV, 1 / 16, kt, vt)
        dims = slice(37, 38) if vt == F16 else slice(32, 64)
        vn[1, dims] = 1e6
        want[0, 6:12, dims] = np.inf
        dk, dv, dkn, dvn = G.dev(kc), G.dev(vc), G.dev(kn), G.dev(vn)
        rd.check(lib.rd_attn_decode_append_ws(rd.ptr(dq), rd.ptr(dkn), rd.ptr(dvn), rd.ptr(dk), rd.ptr(dv), rd.ptr(out),
                                              n - 1, NH, NKV, HD, 1 / 16, kt, vt, None, rd.ptr(ws), nb, G.st()))
    else:
        plant(vc, want, vt, n - 1, 1, [n - 1])
        dk, dv = G.dev(kc), G.dev(vc)
        rd.check(lib.rd_attn_decode_ws(rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), None, 0, n - 1, NH, NKV, HD,
                                       1 / 16, kt, vt, 1, None, rd.ptr(ws), nb, G.st()))
    torch.cuda.synchronize()
    same(G.host(out), want, f"{n} keys")
    G.status_ok()


@pytest.mark.parametrize("n_q,pos0,splits", [(5, 0, 1), (200, 0, 1), (130, 4000, 4)])
def test_prefill_gate_nan(G, oracle, n_q, pos0, splits):
    """A NaN gate makes its own output NaN, with and without a key split; infinite gates give 0 and the whole value."""
    rd, lib = G.rd, G.lib
    n = pos0 + n_q
    z = C.c_int()
    rd.check(lib.rd_attn_prefill_launch_plan(n_q, n, NH, 148, None, None, C.addressof(z), None))
    assert z.value == splits
    q, kc, vc = make(oracle, n, n, F16, F16, n_q)
    pos = np.arange(pos0, n, dtype=np.int32)
    clean = oracle.attn(q, kc, vc, pos, NKV, 1 / 16, F16, F16)
    gate = np.random.default_rng(2).standard_normal(q.shape).astype(np.float32)
    at = ((0, 0, 0), (0, 3, 17), (n_q - 1, 23, 255), (n_q // 2, 7, 100), (n_q // 2, 7, 102))
    for i in at:
        gate[i] = np.nan
    gate[0, 3, 16], gate[1, 5, 64], gate[1, 5, 65] = np.inf, -np.inf, np.inf
    with np.errstate(over="ignore"):
        want = clean * (1 / (1 + np.exp(-gate)))
    dq, dk, dv, dg, dp, out = G.dev(q), G.dev(kc), G.dev(vc), G.dev(gate), G.dev(pos), G.poison(q.shape)
    rd.check(lib.rd_attn_prefill_fused(rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), rd.ptr(dg), rd.ptr(dp), n_q, n, NH,
                                       NKV, HD, 1 / 16, 0, 0.0, G.st()))
    torch.cuda.synchronize()
    same(G.host(out), want, f"{n_q} at {pos0}")
    G.status_ok()


def test_balanced_prefill_parts_without_keys_of_a_row(G):
    """A tile's first token attends all keys, the others the first 100 at most: an infinite row behind those lies in parts
    of the tile's keys that they have nothing in, and is added to no output of theirs. Against f64."""
    rd, lib = G.rd, G.lib
    n_q, n = 450, 9450
    tokens, z = C.c_int(), C.c_int()
    rd.check(lib.rd_attn_prefill_launch_plan(n_q, n, NH, 148, None, C.addressof(tokens), C.addressof(z), None))
    assert (tokens.value, z.value) == (42, 0)
    g = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randn(n_q, NH, HD, device="cuda", generator=g)
    K, V = (torch.randn(n, NKV, HD, device="cuda", generator=g).half() for _ in range(2))
    V[n - 3, :, 5] = torch.inf
    pos = torch.randint(0, 100, (n_q,), dtype=torch.int32, device="cuda", generator=g)
    pos[::42], pos[7] = n - 1, -1
    out = torch.full_like(q, float("nan"))
    rd.check(lib.rd_fa2_prefill(rd.ptr(q), rd.ptr(K), rd.ptr(V), rd.ptr(out), rd.ptr(pos), n_q, n - 1, n, NH, NKV, HD, 1 / 16,
                                G.st()))
    torch.cuda.synchronize()
    G.status_ok()
    past, V[n - 3, :, 5] = torch.arange(n, device="cuda")[None, :] > pos[:, None], 0
    for h in range(NH):
        s = (q[:, h].double() @ K[:, h // 6].double().T / 16).masked_fill_(past, -torch.inf)
        want = torch.nan_to_num(torch.softmax(s, 1)) @ V[:, h // 6].double()
        want[::42, 5] = torch.inf
        same(out[:, h].cpu().numpy(), want.cpu().numpy(), f"head {h}")
