"""fp32 results against 64 bits, as relative 2-norms: what the products' order and unit leave of them.

Sums of up to 64 products in plain fp32 end within sqrt(64) roundings of 2^-24 in either direction, 2.4e-7 and half of that as
a 2-norm over many results;  three TF32 passes end at 4.6e-7 and more."""
import pytest
import torch

import workloads
from oracle import formula

pytestmark = pytest.mark.gpu
DEV = "cuda"
PLAIN = 2.4e-7


def _norm_err(x, want):
    return ((x.double() - want).norm() / want.norm()).item()


def _step(kind, b, h, n, m, seed):
    """({name: error}) of a forward and backward pass of QK and AV"""
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction
    idx = workloads.make_index(kind, b, n, m, seed, DEV)
    g = torch.Generator(device=DEV).manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    q, k, v, g_feat = (rn(b, h, n, 32) for _ in range(4))
    attn, g_attn = torch.softmax(rn(b, h, n, m), -1), rn(b, h, n, m)
    leaf = [t.requires_grad_(True) for t in (q, k, attn, v)]
    out = CLUSTENQKFunction.apply(q, k, idx), CLUSTENAVFunction.apply(attn, v, idx)
    got = out + torch.autograd.grad(out, leaf, (g_attn, g_feat))
    d = [t.detach().double() for t in leaf]
    a, dq, dk = formula.forward_backward("qk", d[0], d[1], idx, g_attn.double(), chunk=1)
    f, da, dv = formula.forward_backward("av", d[2], d[3], idx, g_feat.double(), chunk=1)
    return {name: _norm_err(x, w) for name, x, w in zip(("attn", "feat", "d_query", "d_key", "d_attn", "d_value"), got, (a, f, dq, dk, da, dv))}


@pytest.mark.parametrize("kind,n,m", [("shared", 49, 49), ("shared", 64, 64), ("random", 500, 60)])
def test_rows_of_more_than_48(lib, kind, n, m):
    err = _step(kind, 4, 8, n, m, 800)
    assert max(err[k] for k in ("attn", "feat", "d_query", "d_attn")) <= PLAIN, err


@pytest.mark.parametrize("n,m", [(1000, 48), (500, 40), (300, 13)])
def test_sums_over_rows_of_their_own(lib, n, m):
    """Tables without locality: d_query and the forward of AV."""
    err = _step("random", 4, 4, n, m, 810)
    assert max(err[k] for k in ("feat", "d_query")) <= PLAIN, err


# d_key and d_value over whole clusters, three TF32 passes: errors of the kernels that added up 48 rows at a time
@pytest.mark.parametrize("b,h,n,limit", [(8, 8, 196, 6.4e-7), (4, 8, 1843, 6.6e-7), (8, 2, 3136, 7.1e-7)])
def test_gradients_over_long_lists(lib, b, h, n, limit):
    err = _step("model", b, h, n, 48, 3)
    assert max(err[k] for k in ("d_key", "d_value")) <= 1.02 * limit, err


@pytest.mark.parametrize("b,h,n,m", [(4, 2, 3136, 48), (4, 8, 1843, 48), (4, 4, 784, 24)])
def test_fused_attention_with_a_blank_token(lib, b, h, n, m):
    """The kernel before the online softmax had 9.9e-7 at m = 48, 7.8e-7 at m = 24."""
    from clusten import ops
    idx = workloads.make_index("model", b, n, m, 3, DEV)
    g = torch.Generator(device=DEV).manual_seed(6)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    q, k, v = rn(b, h, n, 32) * 32 ** -0.5, rn(b, h, n, 32), rn(b, h, n, 32)
    table, pe_idx = rn(12321, h), torch.randint(0, 12321, (b, n, m), device=DEV, generator=g)
    blank_k, blank_v = rn(h, 32), rn(h, 32)
    got = ops.local_attention_forward(q, k, v, idx, pe_table=table, pe_idx=pe_idx, blank_k=blank_k, blank_v=blank_v)
    want = []
    for i in range(b):
        logits = formula.qk(q[i:i + 1].double(), k[i:i + 1].double(), idx[i:i + 1])[0] + table.double()[pe_idx[i]].permute(2, 0, 1)
        blank = (q[i].double() * blank_k.double().unsqueeze(1)).sum(-1, keepdim=True)
        p = torch.cat([logits, blank], -1).softmax(-1)
        want.append(formula.av(p[None, ..., :m], v[i:i + 1].double(), idx[i:i + 1])[0] + p[..., m:] * blank_v.double().unsqueeze(1))
    assert _norm_err(got, torch.stack(want)) <= (9.9e-7 if m == 48 else 7.9e-7)
