"""QK / AV on views and over a table's groups: the tables and layouts that the group kernels distinguish -- padded last
clusters, clusters named twice, one list per 8 rows, rows of their own, row counts that are not multiples of the tile --
against the gather formulation in fp64 on the dtype-rounded inputs."""
import pytest
import torch

import workloads
from helpers import TOL, rel_err
from oracle import formula

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _table(kind, b, n, m, seed):
    if kind == "twice":                                   # every third row names its first cluster twice
        idx = workloads.model_like_rows(b, n, m, seed, DEV)
        idx[:, ::3, 8:16] = idx[:, ::3, 0:8]
        return idx
    if kind == "mixed":                                   # a different kind of table per batch element
        return torch.stack([workloads.make_index(k, 1, n, m, seed, DEV)[0] for k in ("model", "shared", "random")])
    if kind == "outside":
        idx = workloads.make_index("shared", b, n, m, seed, DEV)
        idx[:, ::5, 3] = -1
        idx[:, 1::7, m - 1] = n + 2
        return idx
    return workloads.make_index(kind, b, n, m, seed, DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16], ids=["float32", "bfloat16", "float16"])
@pytest.mark.parametrize("kind,n,m", [("model", 17, 16), ("model", 73, 48), ("model", 196, 48), ("model", 1001, 48),
                                      ("model", 64, 8), ("model", 392, 64), ("twice", 203, 48), ("mixed", 200, 48),
                                      ("shared", 49, 49), ("shared", 57, 48), ("outside", 104, 48), ("random", 97, 13),
                                      ("model", 9, 8)])
def test_views_forward_backward(lib, kind, n, m, dtype):
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction, clear_inverse_cache
    b, h, c = 3, 3, 32
    idx = _table(kind, b, n, m, 500 + n)
    g = torch.Generator(device=DEV).manual_seed(501)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)  # noqa: E731
    q = rn(b, n, h * c).view(b, n, h, c).permute(0, 2, 1, 3)
    kv = rn(b, n, 2 * h * c).view(b, n, h, 2, c).permute(3, 0, 2, 1, 4)
    attn, g_attn = rn(b, h, n, m + 1)[..., :-1], rn(b, h, n, m + 1)[..., :-1]
    g_feat = rn(b, n, h, c).permute(0, 2, 1, 3)
    leaf = [t.detach().requires_grad_(True) for t in (q, kv[0], attn, kv[1])]
    out = CLUSTENQKFunction.apply(leaf[0], leaf[1], idx), CLUSTENAVFunction.apply(leaf[2], leaf[3], idx)
    got = out + torch.autograd.grad(out, leaf, (g_attn, g_feat))
    ok = ((idx >= 0) & (idx < n)).double().unsqueeze(1)     # an index outside contributes nothing
    safe = idx.clamp(0, n - 1)
    a, dq, dk = formula.forward_backward("qk", q.double(), kv[0].double(), safe, g_attn.double() * ok)
    f, da, dv = formula.forward_backward("av", attn.double() * ok, kv[1].double(), safe, g_feat.double())
    for name, x, want in zip(("attn", "feat", "d_query", "d_key", "d_attn", "d_value"), got, (a * ok, f, dq, dk, da * ok, dv)):
        assert rel_err(x, want) <= TOL[dtype], name
    clear_inverse_cache()
    again = torch.autograd.grad((CLUSTENQKFunction.apply(leaf[0], leaf[1], idx), CLUSTENAVFunction.apply(leaf[2], leaf[3], idx)), leaf,
                                (g_attn, g_feat))
    assert all(torch.equal(x, y) for x, y in zip(got[2:], again)), "the order of summation is fixed"


@pytest.mark.parametrize("n,m", [(8191, 64), (8184, 64), (9361, 56)])
def test_lists_that_name_a_target_tile_per_slot(lib, n, m):
    """Lists whose slots are 8 tokens apart: as many (list, target tile) pairs as there are slots, at and above what the index of
    the backward pass counts in 16 bits."""
    from clusten import CLUSTENAVFunction
    first = 8 * (torch.arange(n, device=DEV) // 8).view(1, n, 1)
    idx = (first + 8 * torch.arange(m, device=DEV)) % n
    assert (idx[:, :8] == idx[:, :1]).all()
    g = torch.Generator(device=DEV).manual_seed(510)
    attn, v, grad = (torch.randn(1, 1, n, w, generator=g, device=DEV) for w in (m, 32, 32))
    leaf = attn.requires_grad_(True), v.requires_grad_(True)
    got = torch.autograd.grad(CLUSTENAVFunction.apply(*leaf, idx), leaf, grad)
    want = formula.forward_backward("av", attn.detach().double(), v.detach().double(), idx, grad.double())[1:]
    for name, x, w in zip(("d_attn", "d_value"), got, want):
        assert rel_err(x, w) <= TOL[torch.float32], name


@pytest.mark.parametrize("table,message", [(lambda t: t.int(), "int64"), (lambda t: t[0], "3 dimensions"), (lambda t: t.cpu(), "CUDA"),
                                           (lambda t: t[:, :-1].contiguous(), "mismatch")])
def test_tables_that_are_none(lib, table, message):
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction
    idx = table(workloads.make_index("model", 1, 64, 48, 520, DEV))
    q, attn = torch.zeros(1, 2, 64, 32, device=DEV), torch.zeros(1, 2, 64, 48, device=DEV)
    with pytest.raises(RuntimeError, match=message):
        CLUSTENQKFunction.apply(q, q, idx)
    with pytest.raises(RuntimeError, match=message):
        CLUSTENAVFunction.apply(attn, q, idx)


def test_rows_half_a_gigabyte_apart(lib):
    """The row stride is kept in 32 bits; eight rows of it are not."""
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction, ops
    n, m, row = 24, 16, 1 << 28                             # bf16: 2^29 bytes
    idx = (8 * torch.tensor([[1, 2], [2, 0], [0, 1]], device=DEV).repeat_interleave(8, 0).unsqueeze(2) + torch.arange(8, device=DEV)).view(1, n, m)
    g = torch.Generator(device=DEV).manual_seed(530)
    x = torch.randn(1, 1, n, 32, generator=g, device=DEV).bfloat16()
    attn = torch.randn(1, 1, n, m, generator=g, device=DEV).bfloat16()
    far = torch.empty((n - 1) * row + 32, dtype=torch.bfloat16, device=DEV).as_strided((1, 1, n, 32), (32, 32, row, 1)).copy_(x)
    for got, want in ((CLUSTENQKFunction.apply(x, far, idx), CLUSTENQKFunction.apply(x, x, idx)),
                      (CLUSTENAVFunction.apply(attn, far, idx), CLUSTENAVFunction.apply(attn, x, idx)),
                      (ops.local_attention_forward(x, far, far, idx), ops.local_attention_forward(x, x, x, idx))):
        assert torch.equal(got, want)
