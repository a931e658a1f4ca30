"""Decode with a workspace of the records of the all-heads launch and no more (rd_attn_plan's splits): enough for every
length, whichever launch a larger workspace takes; below it the call is refused. Against the oracle."""
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


def record_bytes(rd, n_keys, nkv, kt, vt):
    s = C.c_int()
    rd.check(rd.lib.rd_attn_plan(n_keys, 1, nkv, kt, vt, 0, None, None, C.addressof(s)))
    return 6 * nkv * s.value * (2 + HD) * 4


@pytest.mark.parametrize("append", [False, True])
@pytest.mark.parametrize("kt,vt,nkv,n", [(3, 3, 4, 1), (3, 3, 4, 10), (1, 1, 4, 137), (2, 2, 4, 3000), (1, 1, 1, 1500),
                                         (3, 3, 1, 1000), (4, 5, 2, 2000), (2, 1, 1, 900)])
def test_smallest_workspace(G, oracle, append, kt, vt, nkv, n):
    rd, lib = G.rd, G.lib
    rng = np.random.default_rng(n + nkv)
    K, V = (rng.standard_normal((n, nkv, HD)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((6 * nkv, HD)).astype(np.float32)
    kc, vc = oracle.kv_store_rows(kt, K), oracle.kv_store_rows(vt, V)
    nb = record_bytes(rd, n - 1 if append else n, nkv, kt, vt)
    dq, dk, dv, dkn, dvn = G.dev(q), G.dev(kc), G.dev(vc), G.dev(K[n - 1]), G.dev(V[n - 1])
    if append:
        dk.view(n, -1)[n - 1] = 0
        dv.view(n, -1)[n - 1] = 0

    def call(out, ws, ws_bytes):
        if append:
            return lib.rd_attn_decode_append_ws(rd.ptr(dq), rd.ptr(dkn), rd.ptr(dvn), rd.ptr(dk), rd.ptr(dv), rd.ptr(out),
                                                n - 1, 6 * nkv, nkv, HD, 1 / 16, kt, vt, None, rd.ptr(ws), ws_bytes, G.st())
        return lib.rd_attn_decode_ws(rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), None, 0, n - 1, 6 * nkv, nkv, HD,
                                     1 / 16, kt, vt, 1, None, rd.ptr(ws), ws_bytes, G.st())

    want = oracle.attn(q[None], kc, vc, [n - 1], nkv, 1 / 16, kt, vt)[0]
    ws = torch.full((lib.rd_attn_workspace_bytes(1, 6 * nkv, HD) + 1024,), 0x5A, dtype=torch.uint8, device="cuda")
    for b in (nb, lib.rd_attn_workspace_bytes(1, 6 * nkv, HD)):
        ws.fill_(0x5A)
        out = G.poison(q.shape)
        rd.check(call(out, ws, b))
        torch.cuda.synchronize()
        check_attn(G.host(out), want, what=f"{b} bytes")
        assert bool((ws[b:] == 0x5A).all())
    if append:
        assert np.array_equal(G.host(dk), kc) and np.array_equal(G.host(dv), vc)
    # one record per head is what a call never does without
    assert call(out, ws, 6 * nkv * (2 + HD) * 4 - 1) == rd.ERR_WORKSPACE
    G.status_ok()
