"""Balanced prefill launches through every entry that makes one: the flags of the records are zeroed by a memset
(rd_attn_prefill_fused), by the chunk's append or by the f16 copy of quantized caches, under the tile kernel that reads
them. Against the same attention in f64."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.conftest import check_attn

pytestmark = pytest.mark.gpu
NH, NKV, HD, N_ROT, BASE = 24, 4, 256, 64, 1e7
F16, Q8_0 = 1, 2


@pytest.fixture(scope="module")
def G(cuda):
    from tests import gpu_util
    return gpu_util


def rotated(x, pos):
    f = torch.tensor([BASE ** (-2 * i / N_ROT) for i in range(N_ROT // 2)], dtype=torch.float64).float().cuda()
    a = (pos.float()[:, None, None] * f).double()
    lo, hi, rest = x.double().split([N_ROT // 2, N_ROT // 2, HD - N_ROT], -1)
    return torch.cat([lo * a.cos() - hi * a.sin(), lo * a.sin() + hi * a.cos(), rest], -1)


class Chunk:
    """One call: inputs from a seed, caches of n keys with the chunk's rows from row0 on."""

    def __init__(self, G, entry, n_q, row0, n, pos0, gate, seed):
        self.G, self.entry, self.n_q, self.row0, self.n, self.kt = G, entry, n_q, row0, n, Q8_0 if entry == "typed" else F16
        g = torch.Generator(device="cuda").manual_seed(seed)
        rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
        self.q, self.kn, self.vn = rand(n_q, NH, HD), rand(n_q, NKV, HD), rand(n_q, NKV, HD)
        self.gate = rand(n_q, NH, HD) if gate else None
        self.pos = torch.arange(pos0, pos0 + n_q, dtype=torch.int32, device="cuda")
        self.out = torch.full_like(self.q, float("nan"))
        row = NKV * G.rd.row_bytes(self.kt)
        self.k, self.v = (torch.empty(n, row, dtype=torch.uint8, device="cuda") for _ in range(2))
        for c in (self.k, self.v):
            G.rd.check(G.lib.rd_kv_store_rows(self.kt, G.rd.ptr(rand(n, NKV * HD)), G.rd.ptr(c), n * NKV * HD, G.st()))
        self.ws = None
        if entry == "typed":
            self.nb = G.lib.rd_attn_prefill_workspace_bytes(self.kt, self.kt, n_q, n, NH, NKV, HD)
            self.ws = torch.full((self.nb,), 0xA5, dtype=torch.uint8, device="cuda")

    def run(self):
        rd, lib, p, st = self.G.rd, self.G.lib, self.G.rd.ptr, self.G.rd.stream_ptr()
        shape, rope = (self.n_q, self.n, NH, NKV, HD, 1 / 16), (N_ROT, BASE)
        if self.entry == "append":
            rd.check(lib.rd_attn_prefill_append_fused(p(self.q), p(self.kn), p(self.vn), p(self.k), p(self.v), p(self.out),
                                                      p(self.gate), p(self.pos), self.n_q, self.row0, *shape[1:], *rope, st))
            return
        rd.check(lib.rd_kv_append(self.kt, self.kt, p(self.kn), p(self.vn), p(self.k[self.row0]), p(self.v[self.row0]),
                                  self.n_q, NKV, HD, p(self.pos), *rope, st))
        if self.entry == "fused":
            rd.check(lib.rd_attn_prefill_fused(p(self.q), p(self.k), p(self.v), p(self.out), p(self.gate), p(self.pos),
                                               *shape, *rope, st))
        else:
            rd.check(lib.rd_attn_prefill_typed(p(self.q), p(self.k), p(self.v), p(self.out), p(self.gate), p(self.pos),
                                               *shape, self.kt, self.kt, *rope, p(self.ws), self.nb, st))

    def values(self, cache):
        if self.kt == F16:
            return cache.view(torch.float16).double().view(self.n, NKV, HD)
        b = cache.view(-1, 34)
        x = b[:, 2:].contiguous().view(torch.int8).double() * b[:, :2].contiguous().view(torch.float16).double()
        return x.view(self.n, NKV, HD)

    def check(self, what):
        got, q, K, V = self.out, rotated(self.q, self.pos), self.values(self.k), self.values(self.v)
        past = torch.arange(self.n, device="cuda")[None, :] > self.pos[:, None]
        for h in range(0, NH, 5):
            s = (q[:, h] @ K[:, h // 6].T / 16).masked_fill_(past, -torch.inf)
            want = torch.softmax(s, 1) @ V[:, h // 6]
            if self.gate is not None:
                want *= torch.sigmoid(self.gate[:, h].double())
            a, b = got[:, h].cpu().numpy(), want.cpu().numpy()
            nan = np.isnan(b)   # where the gate is NaN
            assert np.array_equal(np.isnan(a), nan), f"{what} head {h}"
            check_attn(np.where(nan, 0, a), np.where(nan, 0, b), what=f"{what} head {h}")


def assert_balanced(G, n_q, n):
    z = C.c_int()
    G.rd.check(G.lib.rd_attn_prefill_launch_plan(n_q, n, NH, 148, None, None, C.addressof(z), None))
    assert z.value == 0


# a late chunk; tiles of three heads; and positions far below the keys of the call, so that most parts have no key tiles
@pytest.mark.parametrize("n_q,row0,n,pos0", [(512, 7680, 8192, 7680), (389, 11957, 12346, 11957), (389, 40, 12346, 40)])
@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("entry", ["fused", "append", "typed"])
def test_back_to_back(G, entry, gate, n_q, row0, n, pos0):
    """Three layers' calls in a row, each with inputs of its own: flags or records left by the one before would show."""
    assert_balanced(G, n_q, n)
    chunks = [Chunk(G, entry, n_q, row0, n, pos0, gate, seed) for seed in range(3)]
    if entry == "typed":   # layers of one engine share the workspace
        for c in chunks:
            c.ws = chunks[0].ws
    torch.cuda.synchronize()
    for c in chunks:
        c.run()
    torch.cuda.synchronize()
    G.status_ok()
    for i, c in enumerate(chunks):
        c.check(f"call {i}")


@pytest.mark.parametrize("n_q,pos0", [(512, 7680), (389, 11957)])
@pytest.mark.parametrize("entry", ["fused", "append", "typed"])
def test_nan_gate(G, entry, n_q, pos0):
    """A NaN gate makes its own output NaN in the part that collects records, and no other; infinite ones give 0 and 1."""
    assert_balanced(G, n_q, pos0 + n_q)
    c = Chunk(G, entry, n_q, pos0, pos0 + n_q, pos0, True, 7)
    for at in ((0, 0, 0), (0, 5, 17), (n_q - 1, 20, 255), (n_q // 2, 10, 100), (n_q // 2, 10, 102)):
        c.gate[at] = torch.nan
    c.gate[0, 5, 16], c.gate[1, 5, 64], c.gate[1, 5, 65] = torch.inf, -torch.inf, torch.inf
    c.run()
    torch.cuda.synchronize()
    G.status_ok()
    c.check("NaN gate")


@pytest.mark.parametrize("entry", ["fused", "append", "typed"])
def test_captured(G, entry):
    """Captured once, replayed with other inputs in the same buffers."""
    n_q, pos0 = 389, 11957
    assert_balanced(G, n_q, pos0 + n_q)
    c, other = (Chunk(G, entry, n_q, pos0, pos0 + n_q, pos0, True, seed) for seed in (1, 2))
    c.run()   # (grows the library's workspace)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c.run()
    for swap in (False, True, False):
        if swap:
            for x, y in ((c.q, other.q), (c.kn, other.kn), (c.vn, other.vn), (c.gate, other.gate), (c.k, other.k), (c.v, other.v)):
                x.copy_(y)
        c.out.fill_(float("nan"))
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        c.check(f"replay, other inputs {swap}")
    G.status_ok()
