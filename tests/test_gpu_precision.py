"""Error against 64 bits (2-norm over the 2-norm of the result) over f16 caches of normal values.

Weights reach the tensor cores as f16: where the softmax reference is a key's own score its weight is exactly 1.
The bounds are what a kernel with one reference per run of 16 keys (and, for the longer ones, per split) was measured
to give on these inputs, so that longer runs do not cost precision. Rounding the queries alone gives 2.0e-4."""
import pytest
import torch

pytestmark = pytest.mark.gpu
NKV, NH, HD = 4, 24, 256


@pytest.fixture(scope="module")
def G(cuda):
    from tests import gpu_util
    return gpu_util


def exact(q, k, v, pos):
    """q [n_tok][NH][HD], caches [n][NKV][HD], all f64."""
    out = []
    for qi, t in zip(q, pos):
        s = torch.einsum("ghd,ngd->ghn", qi.view(NKV, 6, HD), k[:t + 1]) / 16
        out.append(torch.einsum("ghn,ngd->ghd", torch.softmax(s, -1), v[:t + 1]).reshape(NH, HD))
    return torch.stack(out)


# tokens, keys, bound, what it was with longer runs
@pytest.mark.parametrize("n_tok,n,bound", [(1, 137, 2.52e-4), (1, 3000, 2.58e-4), (1, 4096, 2.60e-4),   # 2.45 2.69 2.76e-4
                                           (2, 100, 2.36e-4), (4, 1000, 2.55e-4), (5, 4096, 2.88e-4),   # 2.75 2.99 2.97e-4
                                           (5, 20011, 2.95e-4), (8, 20011, 2.96e-4)])                   # 2.96 2.96e-4
def test_error_against_64_bits(G, n_tok, n, bound):
    rd, lib = G.rd, G.lib
    errs = []
    for seed in (1, 2, 3):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed * 1000 + n)
        k, v = (torch.randn(n, NKV, HD, device="cuda", generator=g).half() for _ in range(2))
        q = torch.randn(n_tok, NH, HD, device="cuda", generator=g)
        out, pos = G.poison(q.shape), torch.arange(n - n_tok, n, dtype=torch.int32, device="cuda")
        if n_tok == 1:
            rc = lib.rd_attn_decode(rd.ptr(q), rd.ptr(k), rd.ptr(v), rd.ptr(out), n - 1, NH, NKV, HD, 1 / 16, 1, 1, G.st())
        else:
            rc = lib.rd_attn_batch(rd.ptr(q), rd.ptr(k), rd.ptr(v), rd.ptr(out), rd.ptr(pos), n_tok, NH, NKV, HD, 1 / 16,
                                   1, 1, G.st())
        rd.check(rc)
        want = exact(q.double(), k.double(), v.double(), pos.tolist())
        errs.append(float((out.double() - want).norm() / want.norm()))
    assert sum(errs) / 3 <= bound, errs
    G.status_ok()
