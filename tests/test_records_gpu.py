"""Records of a neighbour table's tiles (csrc/group_core.cuh): what they say about rows that are one list of 8k slots, k odd, and
the operators over them.  The operands lie inside larger buffers of NaN, so that a row read from elsewhere shows."""
import pytest
import torch

import workloads
from helpers import TOL, rel_err
from oracle import formula

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inside(t, pad=1024):
    """t as a part of a larger buffer of NaN, `pad` rows around it"""
    flat = t.reshape(-1)
    big = torch.full((flat.numel() + 2 * pad * 32,), float("nan"), dtype=t.dtype, device=t.device)
    big[pad * 32:pad * 32 + flat.numel()] = flat
    return big[pad * 32:pad * 32 + flat.numel()].view(t.shape)


def _sources(idx, n):
    """(kind, list entries) of every tile's record"""
    from clusten import ops
    tiles = idx.shape[0] * ((idx.shape[1] + 15) // 16)
    rec = ops.build_groups(idx, n)[:tiles * 128].view(tiles, 128)
    return rec[:, 0] & 0xff, (rec[:, 16:80].contiguous().view(torch.int16).int() & 0xffff).view(tiles, 2, 64)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16], ids=["float32", "bfloat16", "float16"])
@pytest.mark.parametrize("clusters", [(0, 0, 1), (3, 1, 3, 2, 0), (2,), (5, 5, 4, 3, 2, 1, 5)])
@pytest.mark.parametrize("n", [64, 49])
def test_one_list_with_an_odd_number_of_groups(lib, clusters, n, dtype):
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction, ops
    b, h, m = 1, 2, 8 * len(clusters)
    row = torch.cat([torch.arange(8 * c, 8 * c + 8) for c in clusters])
    idx = row.view(1, 1, m).expand(b, n, m).contiguous().to(DEV)
    kind, sources = _sources(idx, n)
    assert ((sources < n) | (sources == 0xffff) | (kind != 1).view(-1, 1, 1)).all(), "a source row that does not exist"
    g = torch.Generator(device=DEV).manual_seed(601)
    rn = lambda *s: _inside(torch.randn(*s, generator=g, device=DEV).to(dtype))  # noqa: E731
    q, k, v, g_feat = (rn(b, h, n, 32) for _ in range(4))
    attn, g_attn = rn(b, h, n, m), rn(b, h, n, m)
    leaf = [t.detach().requires_grad_(True) for t in (q, k, attn, v)]
    out = CLUSTENQKFunction.apply(leaf[0], leaf[1], idx), CLUSTENAVFunction.apply(leaf[2], leaf[3], idx)
    got = out + torch.autograd.grad(out, leaf, (g_attn, g_feat))
    want = [*formula.forward_backward("qk", q.double(), k.double(), idx, g_attn.double()),
            *formula.forward_backward("av", attn.double(), v.double(), idx, g_feat.double())]
    for name, x, w in zip(("attn", "feat", "d_query", "d_key", "d_attn", "d_value"), got, (want[i] for i in (0, 3, 1, 2, 4, 5))):
        assert torch.isfinite(x).all() and rel_err(x, w) <= TOL[dtype], name
    if m <= 48:
        fused = ops.local_attention_forward(q, k, v, idx)
        assert torch.isfinite(fused).all()
        assert rel_err(fused, formula.av(formula.qk(q.double(), k.double(), idx).softmax(-1), v.double(), idx)) <= TOL[dtype], "fused"


def test_clusters_far_apart(lib):
    """Tables of many tokens: neighbours lie far apart along the curve that numbers the tokens.  Whole clusters stay whole
    clusters, also when two of a tile's share a tag (their ids are 1024 apart)."""
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction
    n, h, m = 20000, 1, 48
    idx = workloads.make_index("model", 1, n, m, 610, DEV)
    assert (_sources(idx, n)[0] == 0).float().mean() > 0.99
    idx[:, 160:192] = (idx[:, 160:192] // 8 % 800 + 1024 * (torch.arange(m, device=DEV) // 8 % 2)) * 8 + torch.arange(m, device=DEV) % 8
    idx[:, 320:352] = (torch.tensor([7, 7 + 1024, 9, 9 + 1024, 11, 12], device=DEV).repeat_interleave(8) * 8 + torch.arange(m, device=DEV) % 8)
    g = torch.Generator(device=DEV).manual_seed(611)
    q, k, v, g_feat = (torch.randn(1, h, n, 32, generator=g, device=DEV) for _ in range(4))
    attn, g_attn = (torch.randn(1, h, n, m, generator=g, device=DEV) for _ in range(2))
    leaf = [t.requires_grad_(True) for t in (q, k, attn, v)]
    out = CLUSTENQKFunction.apply(q, k, idx), CLUSTENAVFunction.apply(attn, v, idx)
    got = out + torch.autograd.grad(out, leaf, (g_attn, g_feat))
    d = [t.detach().double() for t in leaf]
    a, dq, dk = formula.forward_backward("qk", d[0], d[1], idx, g_attn.double())
    f, da, dv = formula.forward_backward("av", d[2], d[3], idx, g_feat.double())
    for name, x, w in zip(("attn", "feat", "d_query", "d_key", "d_attn", "d_value"), got, (a, f, dq, dk, da, dv)):
        assert rel_err(x, w) <= TOL[torch.float32], name


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["float32", "bfloat16"])
@pytest.mark.parametrize("n", [3136, 1001])
def test_tokens_that_a_tile_does_not_name(lib, n, dtype):
    """Values that are not finite stay with the tiles of 16 rows that name them; an odd number of clusters is padded with the
    tile's own."""
    from clusten import CLUSTENAVFunction, ops
    idx = workloads.make_index("model", 1, n, 48, 620, DEV)
    g = torch.Generator(device=DEV).manual_seed(621)
    attn, v, q = (torch.randn(1, 2, n, w, generator=g, device=DEV).to(dtype) for w in (48, 32, 32))
    v[:, :, :8] = float("nan")
    named = torch.zeros(16 * ((n + 15) // 16), dtype=torch.bool, device=DEV)
    named[:n] = (idx[0] < 8).any(1)
    clean = ~named.view(-1, 16).any(1, keepdim=True).expand(-1, 16).reshape(-1)[:n]
    assert clean.float().mean() > 0.5
    assert torch.isfinite(CLUSTENAVFunction.apply(attn, v, idx)[:, :, clean]).all()
    assert torch.isfinite(ops.local_attention_forward(q, q, v, idx)[:, :, clean]).all()
    assert torch.isfinite(ops.local_attention_forward(q, v, q, idx)[:, :, clean]).all()
