"""Blocks of tokens (one CTA per KV head, up to eight tokens): chunk, column-tile and slot edges, fewer KV
heads, ragged positions, records; many sequences with few and many records per row; against the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.conftest import check_attn

pytestmark = pytest.mark.gpu
HD = 256


@pytest.fixture(scope="module")
def G(cuda):
    from tests import gpu_util
    return gpu_util


def make(oracle, seed, nkv, n, kt, vt, n_tok):
    rng = np.random.default_rng(seed)
    K, V = (rng.standard_normal((n, nkv, HD)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((n_tok, 6 * nkv, HD)).astype(np.float32)
    return rng, q, oracle.kv_store_rows(kt, K), oracle.kv_store_rows(vt, V)


@pytest.mark.parametrize("n_tok", [2, 3, 5, 6, 8, 9, 17])
@pytest.mark.parametrize("kt,vt,nkv", [(3, 3, 4), (2, 1, 4), (1, 1, 2), (4, 5, 1), (5, 4, 4), (0, 2, 1)])
def test_block_edges(G, oracle, n_tok, kt, vt, nkv):
    for n in (n_tok, 63, 64, 65, 129, 700):
        n = max(n, n_tok)
        _, q, kc, vc = make(oracle, 7 * n_tok + n, nkv, n, kt, vt, n_tok)
        pos = np.arange(n - n_tok, n, dtype=np.int32)
        want = oracle.attn(q, kc, vc, pos, nkv, 1 / 16, kt, vt)
        check_attn(G.attn_batch(q, kc, vc, pos, kt, vt, nkv=nkv, n_splits=4), want, what=f"{n_tok} tokens, {n} keys")
    G.status_ok()


def test_block_ragged_positions(G, oracle):
    n, nkv = 500, 4
    _, q, kc, vc = make(oracle, 3, nkv, n, 2, 2, 7)
    pos = np.array([499, 0, 64, 63, 128, 17, 320], dtype=np.int32)
    check_attn(G.attn_batch(q, kc, vc, pos, 2, 2), oracle.attn(q, kc, vc, pos, nkv, 1 / 16, 2, 2))


@pytest.mark.parametrize("n_seq,lo,hi,q_len", [(1, 9000, 9001, 1), (2, 5000, 6000, 1), (6, 1500, 4000, 1), (70, 3, 90, 1),
                                               (1, 4000, 4001, 3), (5, 10, 900, 5), (40, 9, 80, 9)])
def test_many_sequences_items_and_merges(G, oracle, n_seq, lo, hi, q_len):
    """One record per row up to a hundred of them; plans in kernel parameters and beyond their size."""
    rd, lib = G.rd, G.lib
    kt, vt, nkv, nh = 3, 2, 4, 24
    rng = np.random.default_rng(n_seq + q_len)
    lens = rng.integers(lo, hi, size=n_seq)
    seqs, keep = (rd.AttnSeq * n_seq)(), []
    for i, n in enumerate(lens):
        n = max(int(n), q_len)
        _, q, kc, vc = make(oracle, 100 + i, nkv, n, kt, vt, q_len)
        gate = rng.standard_normal(q.shape).astype(np.float32)
        dq, dk, dv, dg, out = G.dev(q), G.dev(kc), G.dev(vc), G.dev(gate), G.poison(q.shape)
        seqs[i].q, seqs[i].k, seqs[i].v, seqs[i].out = rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out)
        seqs[i].gate, seqs[i].t = rd.ptr(dg), n - 1
        keep.append((dq, dk, dv, dg, out, q, kc, vc, gate, n))
    nb = lib.rd_attn_multi_workspace_bytes(n_seq, q_len, nh, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        for k in keep:
            k[3].copy_(torch.from_numpy(k[8]))
        rd.check(lib.rd_attn_decode_multi(C.addressof(seqs), n_seq, q_len, nh, nkv, HD, 1 / 16, kt, vt, rd.ptr(ws), nb,
                                          G.st()))
    torch.cuda.synchronize()
    for i in range(0, n_seq, max(1, n_seq // 6)):
        dq, dk, dv, dg, out, q, kc, vc, gate, n = keep[i]
        want = oracle.attn(q, kc, vc, np.arange(n - q_len, n, dtype=np.int32), nkv, 1 / 16, kt, vt)
        sg, want = oracle.sigmoid_gate(gate, want)
        check_attn(G.host(out), want, what=f"sequence {i}, {n} keys")
        assert np.allclose(G.host(dg), sg, atol=1e-6)
    G.status_ok()


# the 64-key slots of a run where many sequences go from two teams of warps to three: 16 (several slots in a team's ring),
# with a single slot 28 in more than a wave of CTAs and 80 in less (four tokens are split again there)
RUNS = [(3, 3, 37, 15), (3, 3, 37, 16), (4, 5, 37, 16), (2, 1, 64, 27), (2, 1, 64, 28), (1, 1, 64, 28), (2, 1, 37, 79),
        (2, 1, 37, 80)]


@pytest.mark.parametrize("kt,vt,n_seq,slots,q_len", [(*r, q) for r in RUNS for q in (2, 4, 5) if (r[3], q) != (80, 4)])
def test_teams_of_many_sequences(G, oracle, kt, vt, n_seq, slots, q_len):
    rd, lib, nkv, nh = G.rd, G.lib, 4, 24
    lens = [64 * slots - i % 3 for i in range(n_seq)]
    t, split = (C.c_int32 * n_seq)(*[n - 1 for n in lens]), (C.c_int32 * n_seq)()
    rd.check(lib.rd_attn_multi_split(C.addressof(t), n_seq, q_len, nkv, kt, vt, 148, C.addressof(split)))
    assert list(split) == [1] * n_seq
    g = torch.Generator(device="cuda").manual_seed(slots + q_len)
    seqs, keep = (rd.AttnSeq * n_seq)(), []
    for i, n in enumerate(lens):
        q, out, caches = torch.randn(q_len, nh, HD, device="cuda", generator=g), G.poison((q_len, nh, HD)), []
        for kind in (kt, vt):
            c = torch.empty(n, nkv * rd.row_bytes(kind), dtype=torch.uint8, device="cuda")
            rd.check(lib.rd_kv_store_rows(kind, rd.ptr(torch.randn(n, nkv * HD, device="cuda", generator=g)), rd.ptr(c),
                                          n * nkv * HD, G.st()))
            caches.append(c)
        seqs[i].q, seqs[i].k, seqs[i].v, seqs[i].out = rd.ptr(q), rd.ptr(caches[0]), rd.ptr(caches[1]), rd.ptr(out)
        seqs[i].gate, seqs[i].t = None, n - 1
        keep.append((q, *caches, out, n))
    nb = lib.rd_attn_multi_workspace_bytes(n_seq, q_len, nh, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    rd.check(lib.rd_attn_decode_multi(C.addressof(seqs), n_seq, q_len, nh, nkv, HD, 1 / 16, kt, vt, rd.ptr(ws), nb, G.st()))
    torch.cuda.synchronize()
    G.status_ok()
    for i in (0, 1, n_seq - 1):
        q, kc, vc, out, n = keep[i]
        want = oracle.attn(G.host(q), G.host(kc), G.host(vc), np.arange(n - q_len, n, dtype=np.int32), nkv, 1 / 16, kt, vt)
        check_attn(G.host(out), want, what=f"sequence {i}")
