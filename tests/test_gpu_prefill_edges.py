"""Prefill tile kernel: rotary sizes, ragged token tiles with and without gate, key splits, both caches
quantized, fewer KV heads; against the oracle."""
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


def rotated(oracle, x, n_rot, pos):
    """Split-half pairs of the first n_rot dims, in f64."""
    y = x.astype(np.float64).copy()
    h = n_rot // 2
    f = 1e7 ** (-2.0 * np.arange(h) / n_rot)
    a = (pos[:, None] * f.astype(np.float32)).astype(np.float32).astype(np.float64)[:, None, :]
    y[..., :h] = x[..., :h] * np.cos(a) - x[..., h:n_rot] * np.sin(a)
    y[..., h:n_rot] = x[..., :h] * np.sin(a) + x[..., h:n_rot] * np.cos(a)
    return y.astype(np.float32)


@pytest.mark.parametrize("n_rot", [0, 16, 32, 48, 64])
@pytest.mark.parametrize("n_q,pos0,nkv", [(1, 0, 4), (127, 5, 1), (129, 130, 2), (40, 2100, 1), (256, 0, 4)])
def test_rotary_sizes_and_ragged_tiles(G, oracle, n_rot, n_q, pos0, nkv):
    rd, lib = G.rd, G.lib
    n, nh = pos0 + n_q, 6 * nkv
    rng = np.random.default_rng(n_rot + n_q)
    K, V = (rng.standard_normal((n, nkv, HD)).astype(np.float32) for _ in range(2))
    q, gate = (rng.standard_normal((n_q, nh, HD)).astype(np.float32) for _ in range(2))
    pos = np.arange(pos0, n, dtype=np.int32)
    kc, vc = oracle.kv_store_rows(1, K), oracle.kv_store_rows(1, V)
    want = oracle.attn(rotated(oracle, q, n_rot, pos) if n_rot else q, kc, vc, pos, nkv, 1 / 16, 1, 1)
    dq, dk, dv, dpos, dg = G.dev(q), G.dev(kc), G.dev(vc), G.dev(pos), G.dev(gate)
    for g in (None, dg):
        out = G.poison(q.shape)
        rd.check(lib.rd_attn_prefill_fused(rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), rd.ptr(g), rd.ptr(dpos), n_q, n,
                                           nh, nkv, HD, 1 / 16, n_rot, 1e7, G.st()))
        torch.cuda.synchronize()
        check_attn(G.host(out), want if g is None else want / (1 + np.exp(-gate)), what=f"gate {g is not None}")
    G.status_ok()


@pytest.mark.parametrize("n_q,pos0", [(3, 4000), (130, 9000)])
def test_key_splits_of_quantized_caches(G, oracle, n_q, pos0):
    rd, lib = G.rd, G.lib
    nkv, nh, n, kt, vt = 1, 6, pos0 + n_q, 2, 3
    rng = np.random.default_rng(n_q)
    K, V = (rng.standard_normal((n, nkv, HD)).astype(np.float32) for _ in range(2))
    q, gate = (rng.standard_normal((n_q, nh, HD)).astype(np.float32) for _ in range(2))
    pos = np.arange(pos0, n, dtype=np.int32)
    kc, vc = oracle.kv_store_rows(kt, K), oracle.kv_store_rows(vt, V)
    nb = lib.rd_attn_prefill_workspace_bytes(kt, vt, n_q, n, nh, nkv, HD)
    ws, out = torch.empty(nb, dtype=torch.uint8, device="cuda"), G.poison(q.shape)
    dq, dk, dv, dpos, dg = G.dev(q), G.dev(kc), G.dev(vc), G.dev(pos), G.dev(gate)
    rd.check(lib.rd_attn_prefill_typed(rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), rd.ptr(dg), rd.ptr(dpos), n_q, n, nh,
                                       nkv, HD, 1 / 16, kt, vt, 64, 1e7, rd.ptr(ws), nb, G.st()))
    torch.cuda.synchronize()
    want = oracle.attn(rotated(oracle, q, 64, pos), kc, vc, pos, nkv, 1 / 16, kt, vt) / (1 + np.exp(-gate))
    check_attn(G.host(out), want)
    G.status_ok()
