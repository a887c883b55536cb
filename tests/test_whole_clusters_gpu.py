"""QK and AV over whole clusters in 16 bits, forward and backward: blocks of 64 rows with few and with many distinct clusters, blocks
that are not full, lists of rows of every length (none, less than a step, several steps), padded slots, weights that start on
16-byte boundaries and anywhere."""
import pytest
import torch

import workloads
from helpers import TOL, rel_err
from oracle import formula

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bfloat16", "float16"])
@pytest.mark.parametrize("layout", ["plain", "views"])
@pytest.mark.parametrize("b,h,n,groups", [(1, 1, 16, 1), (2, 3, 17, 2), (1, 2, 23, 2), (2, 5, 133, 6), (1, 4, 260, 8), (1, 9, 1037, 3), (2, 2, 320, 6)])
def test_lists_of_every_length(lib, b, h, n, groups, layout, dtype):
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction
    k, m = (n + 7) // 8, 8 * groups
    g = torch.Generator(device=DEV).manual_seed(700 + n)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)  # noqa: E731
    # distinct clusters per row, low ids far more often than high ones, so that some clusters are named by nobody;  the padded one by many
    score = torch.rand(b, n, k, generator=g, device=DEV) + 2.0 * torch.arange(k, device=DEV) / k
    score[:, ::3, -1] = -1.0
    idx = (8 * score.topk(groups, dim=2, largest=False)[1].unsqueeze(3) + torch.arange(8, device=DEV)).view(b, n, m)
    idx[idx >= n] = 0
    if layout == "views":
        q, g_feat = (rn(b, n, h, 32).permute(0, 2, 1, 3) for _ in range(2))
        attn, g_attn = rn(b, h, n, m + 1)[..., 1:], rn(b, h, n, m + 1)[..., :-1]
    else:
        q, g_feat, attn, g_attn = rn(b, h, n, 32), rn(b, h, n, 32), rn(b, h, n, m), rn(b, h, n, m)
    key, v = rn(b, h, n, 32), rn(b, h, n, 32)
    leaf = [t.detach().requires_grad_(True) for t in (q, key, attn, v)]
    out = CLUSTENQKFunction.apply(leaf[0], leaf[1], idx), CLUSTENAVFunction.apply(leaf[2], leaf[3], idx)
    got = out + torch.autograd.grad(out, leaf, (g_attn, g_feat))
    a, dq, dk = formula.forward_backward("qk", q.double(), key.double(), idx, g_attn.double())
    f, da, dv = formula.forward_backward("av", attn.double(), v.double(), idx, g_feat.double())
    for name, x, w in zip(("attn", "feat", "d_query", "d_key", "d_attn", "d_value"), got, (a, f, dq, dk, da, dv)):
        assert rel_err(x, w) <= TOL[dtype], name


@pytest.mark.parametrize("n", [64993, 65000])
def test_clusters_of_many_tokens(lib, n):
    """The forward passes at the largest token counts, rows of 24: a tile's clusters span all ids."""
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction
    k, m = (n + 7) // 8, 24
    first = (torch.arange(n, device=DEV) // 8).view(1, n, 1) + torch.tensor([0, 5, 4001], device=DEV)
    idx = (8 * (first % k).unsqueeze(3) + torch.arange(8, device=DEV)).view(1, n, m)
    idx[idx >= n] = 0
    g = torch.Generator(device=DEV).manual_seed(720)
    q, key, attn = (torch.randn(1, 1, n, w, generator=g, device=DEV).bfloat16() for w in (32, 32, m))
    for got, want in ((CLUSTENQKFunction.apply(q, key, idx), formula.qk(q.double(), key.double(), idx)),
                      (CLUSTENAVFunction.apply(attn, key, idx), formula.av(attn.double(), key.double(), idx))):
        assert rel_err(got, want) <= TOL[torch.bfloat16]


NAMES = ("attn", "feat", "d_query", "d_key", "d_attn", "d_value")


def _operands(b, h, n, m, layout, dtype, seed):
    """query, key, attn, value, d_attn, d_feat;  views: attn and its gradient start anywhere"""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)  # noqa: E731
    if layout == "views":
        q, g_feat = (rn(b, n, h, 32).permute(0, 2, 1, 3) for _ in range(2))
        kv = rn(b, n, h, 2, 32).permute(3, 0, 2, 1, 4)
        return q, kv[0], rn(b, h, n, m + 1)[..., 1:], kv[1], rn(b, h, n, m + 1)[..., :-1], g_feat
    return rn(b, h, n, 32), rn(b, h, n, 32), rn(b, h, n, m), rn(b, h, n, 32), rn(b, h, n, m), rn(b, h, n, 32)


def _train(operands, idx):
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction
    q, k, attn, v, g_attn, g_feat = operands
    leaf = [t.detach().requires_grad_(True) for t in (q, k, attn, v)]
    out = CLUSTENQKFunction.apply(leaf[0], leaf[1], idx), CLUSTENAVFunction.apply(leaf[2], leaf[3], idx)
    return [t.detach() for t in out + torch.autograd.grad(out, leaf, (g_attn, g_feat))]


def _wanted(operands, idx, element):
    q, k, attn, v, g_attn, g_feat = (t[element:element + 1].double() for t in operands)
    table = idx[element:element + 1]
    a, dq, dk = formula.forward_backward("qk", q, k, table, g_attn)
    f, da, dv = formula.forward_backward("av", attn, v, table, g_feat)
    return a, f, dq, dk, da, dv


def _table(kind, b, n, m, seed):
    if kind == "unnamed":                                     # every row names one of the first clusters and the padded one, most are named by nobody
        g = torch.Generator(device=DEV).manual_seed(seed)
        k = (n + 7) // 8
        score = torch.rand(b, n, k, generator=g, device=DEV) + (torch.arange(k, device=DEV) >= m // 8 + 2)
        score[:, ::3, -1] = -1.0
        idx = (8 * score.topk(m // 8, dim=2, largest=False)[1].unsqueeze(3) + torch.arange(8, device=DEV)).view(b, n, m)
        return torch.where(idx < n, idx, 0)
    return workloads.make_index(kind, b, n, m, seed, DEV)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bfloat16", "float16"])
@pytest.mark.parametrize("layout", ["plain", "views"])
@pytest.mark.parametrize("kind,b,h,n,m", [("model", 256, 7, 196, 48), ("model", 256, 2, 196, 48), ("model", 128, 8, 196, 48), ("model", 40, 8, 1843, 48),
                                          ("shared", 256, 7, 196, 48), ("shared", 170, 5, 203, 48), ("unnamed", 256, 7, 201, 48), ("model", 256, 3, 197, 24),
                                          ("shared", 160, 6, 203, 40), ("random", 100, 3, 150, 48)])
def test_several_heads_per_warp(lib, kind, b, h, n, m, layout, dtype):
    """So many tiles that a warp takes two heads and more (148 SMs: 256 batch elements of 7 heads are 4 and 3 to a warp, in gradients and forward)."""
    idx = _table(kind, b, n, m, 730 + n)
    operands = _operands(b, h, n, m, layout, dtype, 731)
    got = _train(operands, idx)
    for element in (0, b // 2 + 1, b - 1):
        for name, x, w in zip(NAMES, got, _wanted(operands, idx, element)):
            assert rel_err(x[element:element + 1], w) <= TOL[dtype], (name, element)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bfloat16", "float16"])
@pytest.mark.parametrize("layout", ["plain", "views"])
def test_blocks_of_many_clusters(lib, layout, dtype):
    """64 rows that name as many clusters as a block holds (40), one more, and far more, while their four tiles have at most 28 each; a last block of
    three tiles, the last one of five rows."""
    from clusten import ops
    b, h, n, m = 12, 16, 1573, 48
    k, tiles = (n + 7) // 8, (n + 15) // 16
    rows = []
    for sizes in ((10, 10, 10, 10), (11, 10, 10, 10), (25, 25, 25, 25)):
        first = torch.tensor([3 * (t // 4) + sum(sizes[:t % 4]) for t in range(tiles)])
        size = torch.tensor([sizes[t % 4] for t in range(tiles)])
        place = (6 * torch.arange(16).view(1, 16, 1) + torch.arange(6)) % size.view(-1, 1, 1)
        rows.append(((first.view(-1, 1, 1) + place) % k).view(-1, 6)[:n])
        assert {len(set(rows[-1][i:i + 64].flatten().tolist())) for i in range(0, n - 63, 64)} == {sum(sizes)}
    idx = (8 * torch.stack(rows).repeat(b // 3, 1, 1).unsqueeze(3) + torch.arange(8)).view(b, n, m)
    idx = torch.where(idx < n, idx, 0).to(DEV)
    assert ((ops.build_groups(idx, n)[:b * tiles * 128].view(-1, 128)[:, 0] & 0xff) == 0).all(), "all tiles have whole clusters"
    operands = _operands(b, h, n, m, layout, dtype, 741)
    got = _train(operands, idx)
    for element in range(3):
        for name, x, w in zip(NAMES, got, _wanted(operands, idx, element)):
            assert rel_err(x[element:element + 1], w) <= TOL[dtype], (name, element)


@pytest.mark.parametrize("n", [64993, 65000])
def test_blocks_of_many_tokens(lib, n):
    """Records and blocks at the largest token counts: the bits of a block's clusters span all ids."""
    from clusten import _lib
    h, k = 5, (n + 7) // 8
    first = (torch.arange(n, device=DEV) // 8).view(1, n, 1) + torch.tensor([0, 5, 4001, k - 9, 2077, 6], device=DEV)
    idx = (8 * (first % k).unsqueeze(3) + torch.arange(8, device=DEV)).view(1, n, 48)
    idx = torch.where(idx < n, idx, 0)
    g = torch.Generator(device=DEV).manual_seed(750)
    q, key, attn = (torch.randn(1, h, n, w, generator=g, device=DEV).bfloat16() for w in (32, 32, 48))
    host = _lib.host()
    for got, fn, x in ((host.qk_forward(q, key, idx, True), formula.qk, q), (host.av_forward(attn, key, idx, True), formula.av, attn)):
        assert got[1] is not None
        for head in (slice(0, 1), slice(4, 5)):
            assert rel_err(got[0][:, head], fn(x[:, head].double(), key[:, head].double(), idx)) <= TOL[torch.bfloat16]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bfloat16", "float16"])
@pytest.mark.parametrize("kind,layout", [("model", "plain"), ("model", "views"), ("shared", "plain")])
def test_values_that_are_not_finite(lib, kind, layout, dtype):
    """A score, and a target's gradient over whole clusters, is not finite where a row that is not takes part, and nowhere else; sums stay finite in
    tiles of 16 rows (lists: of 8 targets) that do not name such a row."""
    b, h, n, m = 40, 8, 1001, 48
    idx = _table(kind, b, n, m, 760)
    operands = _operands(b, h, n, m, layout, dtype, 761)
    q, k, attn, v, g_attn, g_feat = operands
    e = 3
    k[e, :, 400:403], v[e, :, 80:83] = float("nan"), float("inf")
    q[e, :, 17], g_feat[e, :, 300] = float("inf"), float("nan")
    got = _train(operands, idx)
    for name, x in zip(NAMES, got):
        assert torch.isfinite(x[:e]).all() and torch.isfinite(x[e + 1:]).all(), name
    a, f, dq, dk, da, dv = (torch.isfinite(t[0]) for t in _wanted(operands, idx, e))
    ga, gf, gdq, gdk, gda, gdv = (torch.isfinite(t[e]) for t in got)
    assert torch.equal(ga, a) and torch.equal(gda, da)
    tile = lambda t, w: torch.nn.functional.pad(t.all(0).all(1), (0, -n % w), value=True).view(-1, w).all(1).repeat_interleave(w)[:n]  # noqa: E731
    for name, x, w, width in (("feat", gf, f, 16), ("d_query", gdq, dq, 16), ("d_key", gdk, dk, 8), ("d_value", gdv, dv, 8)):
        assert not x[~w].any(), name
        assert x[:, tile(w, width)].all(), name
        if kind == "model" and width == 8:
            assert torch.equal(x, w), name


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bfloat16", "float16"])
@pytest.mark.parametrize("layout", ["plain", "views"])
@pytest.mark.parametrize("kind", ["model", "shared", "random", "unnamed", "outside", "twice", "far"])
@pytest.mark.parametrize("b,h,n", [(8, 16, 2368), (8, 16, 2352), (4, 3, 357), (1, 2, 45)])
def test_over_records_and_without(lib, kind, b, h, n, layout, dtype):
    """Forward passes over records (blocks; dot products from 128 tiles and heads per SM on, 8 x 16 x 148 on 148 SMs) and with records made in the kernel,
    tile by tile: the same products in the same order."""
    from clusten import _lib
    m = 48
    idx = _table(kind if kind in ("model", "shared", "random", "unnamed") else "shared" if kind == "outside" else "model", b, n, m, 770 + n)
    if kind == "outside":
        idx[:, ::5, 3], idx[:, 1::7, m - 1] = -1, n + 2
    elif kind == "twice":                                     # every 37th row names its first cluster twice
        idx[:, ::37, 8:16] = idx[:, ::37, 0:8]
    elif kind == "far":                                       # tiles in any order: blocks of more clusters than they hold, next to others
        tile = torch.arange(n, device=DEV) // 16
        order = torch.where(tile % 8 < 4, tile, (7 * tile + 3) % (n // 16)).clamp_(max=n // 16 - 1)
        idx = idx[:, order * 16 + torch.arange(n, device=DEV) % 16].contiguous()
    q, k, attn, v = _operands(b, h, n, m, layout, dtype, 771)[:4]
    host = _lib.host()
    for over, without in ((host.qk_forward(q, k, idx, True), host.qk_forward(q, k, idx, False)),
                          (host.av_forward(attn, v, idx, True), host.av_forward(attn, v, idx, False))):
        assert over[1] is not None and without[1] is None
        assert torch.equal(over[0], without[0])
