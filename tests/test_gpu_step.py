"""Per-head decode (one cluster per KV head, or records): slot and cluster edges, the lines between the forms,
fewer KV heads, a first key behind 0, the fused append at slot edges; against the oracle."""
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


def make(oracle, seed, nkv, n, kt, vt):
    rng = np.random.default_rng(seed)
    K, V = (rng.standard_normal((n, nkv, HD)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((6 * nkv, HD)).astype(np.float32)
    return rng, q, oracle.kv_store_rows(kt, K), oracle.kv_store_rows(vt, V)


@pytest.mark.parametrize("kt,vt,nkv", [(1, 1, 4), (2, 2, 4), (3, 3, 2), (4, 5, 1), (5, 4, 4), (2, 1, 4), (0, 0, 1)])
def test_short_context_edges(G, oracle, kt, vt, nkv):
    rd, lib = G.rd, G.lib
    n_max = {(2, 2): 8193, (1, 1): 5634, (2, 1): 3586}.get((kt, vt), 1100)
    rng, q, kc, vc = make(oracle, 10 * kt + vt, nkv, n_max, kt, vt)
    gate = rng.standard_normal(q.shape).astype(np.float32)
    dq, dk, dv = G.dev(q), G.dev(kc), G.dev(vc)
    nb = lib.rd_attn_workspace_bytes(1, 6 * nkv, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    for begin, n in ((0, 1), (0, 15), (0, 16), (0, 17), (0, 255), (0, 256), (0, 257), (3, 300), (77, n_max - 1), (0, n_max - 2), (0, n_max)):
        want = oracle.attn(q[None], kc.reshape(n_max, -1)[begin:n], vc.reshape(n_max, -1)[begin:n], [n - begin - 1], nkv,
                           1 / 16, kt, vt)[0]
        sg, want = oracle.sigmoid_gate(gate, want)
        g, out = G.dev(gate), G.poison(q.shape)
        rd.check(lib.rd_attn_decode_ws(rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), None, begin, n - 1, 6 * nkv, nkv,
                                       HD, 1 / 16, kt, vt, 1, rd.ptr(g), rd.ptr(ws), nb, G.st()))
        torch.cuda.synchronize()
        check_attn(G.host(out), want, what=f"keys {begin}..{n - 1}")
        assert np.allclose(G.host(g), sg, atol=1e-6)
    G.status_ok()


@pytest.mark.parametrize("kt,vt", [(1, 1), (3, 3), (4, 5), (2, 1)])
@pytest.mark.parametrize("t", [15, 16, 17, 255, 256, 511, 5700])
def test_short_context_append(G, oracle, kt, vt, t):
    rd, lib = G.rd, G.lib
    nkv = 4
    rng, q, kc, vc = make(oracle, t + 100 * kt, nkv, t + 1, kt, vt)
    kn, vn = (rng.standard_normal((nkv, HD)).astype(np.float32) for _ in range(2))
    k0, v0 = kc.reshape(t + 1, -1).copy(), vc.reshape(t + 1, -1).copy()
    k0[t], v0[t] = oracle.kv_store_rows(kt, kn).reshape(-1), oracle.kv_store_rows(vt, vn).reshape(-1)
    dk, dv = G.dev(kc), G.dev(vc)
    dq, dkn, dvn, out = G.dev(q), G.dev(kn), G.dev(vn), G.poison(q.shape)
    nb = lib.rd_attn_workspace_bytes(1, 24, HD)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    rd.check(lib.rd_attn_decode_append_ws(rd.ptr(dq), rd.ptr(dkn), rd.ptr(dvn), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), t, 24,
                                          nkv, HD, 1 / 16, kt, vt, None, rd.ptr(ws), nb, G.st()))
    torch.cuda.synchronize()
    assert np.array_equal(G.host(dk).reshape(t + 1, -1), k0) and np.array_equal(G.host(dv).reshape(t + 1, -1), v0)
    check_attn(G.host(out), oracle.attn(q[None], k0, v0, [t], nkv, 1 / 16, kt, vt)[0], what=f"append at {t}")
