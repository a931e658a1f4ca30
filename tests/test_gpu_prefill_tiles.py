"""Prefill tiles of three heads x 42 tokens: edges of a tile, rotation, gate, many key splits, a workspace with room
for fewer records than the plan wants; against the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.conftest import check_attn
from tests.test_gpu_prefill_edges import rotated

pytestmark = pytest.mark.gpu
HD, NKV, NH = 256, 1, 6


@pytest.fixture(scope="module")
def G(cuda):
    from tests import gpu_util
    return gpu_util


def plan(lib, n_q, n):
    heads, z = C.c_int(), C.c_int()
    assert lib.rd_attn_prefill_launch_plan(n_q, n, NH, 148, C.addressof(heads), None, C.addressof(z), None) == 0
    return heads.value, z.value


@pytest.mark.parametrize("n_q,pos0,n_rot", [(1, 2100, 64), (31, 2100, 64), (42, 2100, 64), (43, 3000, 64), (64, 3000, 32),
                                            (85, 2100, 64), (126, 2100, 0), (127, 2100, 64), (253, 6000, 64), (24, 9000, 64)])
def test_three_head_tiles(G, oracle, n_q, pos0, n_rot):
    rd, lib = G.rd, G.lib
    n = pos0 + n_q
    heads, z = plan(lib, n_q, n)
    assert heads == 3 and (z > 12 if pos0 == 9000 else z > 1)
    rng = np.random.default_rng(n_q)
    K, V = (rng.standard_normal((n, NKV, HD)).astype(np.float32) for _ in range(2))
    q, gate = (rng.standard_normal((n_q, NH, HD)).astype(np.float32) for _ in range(2))
    pos = np.arange(pos0, n, dtype=np.int32)
    kc, vc = oracle.kv_store_rows(1, K), oracle.kv_store_rows(1, V)
    want = oracle.attn(rotated(oracle, q, n_rot, pos) if n_rot else q, kc, vc, pos, NKV, 1 / 16, 1, 1)
    dq, dk, dv, dpos, dg = G.dev(q), G.dev(kc), G.dev(vc), G.dev(pos), G.dev(gate)
    for g in (None, dg):
        out = G.poison(q.shape)
        rd.check(lib.rd_attn_prefill_fused(rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), rd.ptr(g), rd.ptr(dpos), n_q, n,
                                           NH, NKV, HD, 1 / 16, n_rot, 1e7, G.st()))
        torch.cuda.synchronize()
        check_attn(G.host(out), want if g is None else want / (1 + np.exp(-gate)), what=f"gate {g is not None}")
    G.status_ok()


@pytest.mark.parametrize("n_q,pos0", [(24, 9000), (300, 7000)])
def test_workspace_with_less_room_than_the_plan(G, oracle, n_q, pos0):
    """The records of the plan, those of one-head tiles (what a call has to have), and what lies between."""
    rd, lib = G.rd, G.lib
    n, kt, vt = pos0 + n_q, 2, 2
    rng = np.random.default_rng(n_q)
    K, V = (rng.standard_normal((n, NKV, HD)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((n_q, NH, HD)).astype(np.float32)
    pos = np.arange(pos0, n, dtype=np.int32)
    kc, vc = oracle.kv_store_rows(kt, K), oracle.kv_store_rows(vt, V)
    want = oracle.attn(q, kc, vc, pos, NKV, 1 / 16, kt, vt)
    dq, dk, dv, dpos = G.dev(q), G.dev(kc), G.dev(vc), G.dev(pos)
    full = lib.rd_attn_prefill_workspace_bytes(kt, vt, n_q, n, NH, NKV, HD)
    z = C.c_int()
    rd.check(lib.rd_attn_prefill_plan(n_q, n, NH, 148, C.addressof(z), None))
    align = lambda x: (x + 255) // 256 * 256
    least = 2 * align(n * NKV * HD * 2) + align(n_q * NH * z.value * 1032)
    assert full >= least
    call = lambda out, nb: lib.rd_attn_prefill_typed(rd.ptr(dq), rd.ptr(dk), rd.ptr(dv), rd.ptr(out), None, rd.ptr(dpos), n_q,
                                                     n, NH, NKV, HD, 1 / 16, kt, vt, 0, 0.0, rd.ptr(ws), nb, G.st())
    for nb in sorted({full, (full + least) // 2, least}):
        ws = torch.full((nb + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
        out = G.poison(q.shape)
        rd.check(call(out, nb))
        torch.cuda.synchronize()
        check_attn(G.host(out), want, what=f"{nb} bytes")
        assert (ws[nb:] == 0xA5).all()
    assert call(out, least - 256) == rd.ERR_WORKSPACE
    G.status_ok()


@pytest.mark.parametrize("n_q,n", [(24, 1224), (64, 1864), (200, 1400), (8, 8)])
def test_no_workspace_is_asked_for_that_is_not_used(G, n_q, n):
    """f16 caches whose keys are not split need no workspace, so none is asked for and none is written."""
    rd, lib = G.rd, G.lib
    z = C.c_int()
    rd.check(lib.rd_attn_prefill_plan(n_q, n, 24, 148, C.addressof(z), None))
    assert z.value == 1
    assert lib.rd_attn_prefill_workspace_bytes(1, 1, n_q, n, 24, 4, HD) == 0
    copies = 2 * ((n * 4 * HD * 2 + 255) // 256 * 256)
    assert lib.rd_attn_prefill_workspace_bytes(2, 2, n_q, n, 24, 4, HD) >= copies


@pytest.mark.parametrize("n_q,pos0,heads,nh,ragged", [(389, 11957, 3, 24, False), (512, 7680, 1, 24, False), (1000, 7000, 3, 24, False),
                                                      (450, 9000, 3, 24, True), (2000, 6000, 3, 12, False)])
def test_balanced_launches(G, n_q, pos0, heads, nh, ragged):
    """Parts of key ranges cut anywhere, records collected by the part that writes: against the same attention in f64,
    with positions in order and with ones that the plan did not expect; twice, into the records of the first run."""
    rd, lib = G.rd, G.lib
    n, nkv = pos0 + n_q, nh // 6
    got = [C.c_int() for _ in range(4)]
    rd.check(lib.rd_attn_prefill_launch_plan(n_q, n, nh, 148, *[C.addressof(x) for x in got]))
    assert [x.value for x in got[::2]] == [heads, 0]
    g = torch.Generator(device="cuda").manual_seed(n_q)
    q, gate = (torch.randn(n_q, nh, HD, device="cuda", generator=g) for _ in range(2))
    K, V = (torch.randn(n, nkv, HD, device="cuda", generator=g).half() for _ in range(2))
    pos = torch.arange(pos0, n, dtype=torch.int32, device="cuda")
    if ragged:
        pos = torch.randint(0, n, (n_q,), dtype=torch.int32, device="cuda", generator=g)
        pos[7], pos[300:] = -1, pos[300:] // 8
    out = torch.full_like(q, float("nan"))
    for _ in range(2):
        rd.check(lib.rd_attn_prefill_fused(rd.ptr(q), rd.ptr(K), rd.ptr(V), rd.ptr(out), rd.ptr(gate), rd.ptr(pos), n_q, n, nh,
                                           nkv, HD, 1 / 16, 0, 0.0, G.st()))
    torch.cuda.synchronize()
    G.status_ok()
    past = torch.arange(n, device="cuda")[None, :] > pos[:, None]
    for h in range(0, nh, 5):
        s = (q[:, h].double() @ K[:, h // 6].double().T / 16).masked_fill_(past, -torch.inf)
        want = torch.nan_to_num(torch.softmax(s, 1)) @ V[:, h // 6].double() * torch.sigmoid(gate[:, h].double())
        check_attn(out[:, h].cpu().numpy(), want.cpu().numpy(), what=f"head {h}")
    if ragged:
        assert (out[7] == 0).all()


@pytest.mark.parametrize("n_q,pos0", [(512, 7680), (1000, 7000)])
def test_balanced_launch_reads_the_records_of_its_own_pass(G, n_q, pos0):
    """Two inputs in turn through the same record memory: a value collected before its part had written it is the other
    input's, so every pass has to give the bits that the input gave the first time."""
    rd, lib = G.rd, G.lib
    n, nh, nkv = pos0 + n_q, 24, 4
    z = C.c_int()
    rd.check(lib.rd_attn_prefill_launch_plan(n_q, n, nh, 148, None, None, C.addressof(z), None))
    assert z.value == 0
    g = torch.Generator(device="cuda").manual_seed(n_q)
    pos = torch.arange(pos0, n, dtype=torch.int32, device="cuda")
    inputs = []
    for _ in range(2):
        q = torch.randn(n_q, nh, HD, device="cuda", generator=g)
        K, V = (torch.randn(n, nkv, HD, device="cuda", generator=g).half() for _ in range(2))
        inputs.append((q, K, V, *(torch.randn(n_q, nkv, HD, device="cuda", generator=g) for _ in range(2))))
    out, first = torch.empty_like(inputs[0][0]), [None, None]
    for i in range(24):
        q, K, V, kn, vn = inputs[i & 1]
        rd.check(lib.rd_attn_prefill_append_fused(rd.ptr(q), rd.ptr(kn), rd.ptr(vn), rd.ptr(K), rd.ptr(V), rd.ptr(out), None,
                                                  rd.ptr(pos), n_q, pos0, n, nh, nkv, HD, 1 / 16, 64, 1e7, G.st()))
        if first[i & 1] is None:
            first[i & 1] = out.clone()
        assert torch.equal(out, first[i & 1]), i
    assert not torch.equal(*first)
    G.status_ok()
