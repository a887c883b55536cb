"""QK and AV over whole clusters in 16 bits, forward and backward: blocks of 64 rows with few and with many distinct clusters, blocks
that are not full, lists of rows of every length (none, less than a step, several steps), padded slots, weights that start on
16-byte boundaries and anywhere."""
import pytest
import torch

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
    """The forward passes at the largest token counts: the block's clusters span all ids."""
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
