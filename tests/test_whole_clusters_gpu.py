"""d_key and d_value over whole clusters in 16 bits: lists of every length (none, less than a step, several steps), padded slots,
weights that start on 16-byte boundaries and anywhere."""
import pytest
import torch

from helpers import TOL, rel_err
from oracle import formula

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bfloat16", "float16"])
@pytest.mark.parametrize("layout", ["plain", "views"])
@pytest.mark.parametrize("b,h,n,groups", [(1, 1, 16, 1), (2, 3, 17, 2), (1, 2, 23, 2), (2, 5, 133, 6), (1, 4, 260, 8), (1, 9, 1037, 3)])
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
    key, v = rn(b, h, n, 32).requires_grad_(True), rn(b, h, n, 32).requires_grad_(True)
    out = CLUSTENQKFunction.apply(q, key, idx), CLUSTENAVFunction.apply(attn, v, idx)
    got = torch.autograd.grad(out, (key, v), (g_attn, g_feat))
    want = (formula.forward_backward("qk", q.double(), key.detach().double(), idx, g_attn.double())[2],
            formula.forward_backward("av", attn.double(), v.detach().double(), idx, g_feat.double())[2])
    for name, x, w in zip(("d_key", "d_value"), got, want):
        assert rel_err(x, w) <= TOL[dtype], name
