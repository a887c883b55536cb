"""Buffers that the package derives from a neighbour table, and tables that change: what the operators return follows from the
table's contents at the call."""
import pytest
import torch

import workloads
from helpers import TOL, rel_err
from oracle import formula

pytestmark = pytest.mark.gpu
DEV = "cuda"
SIZES = [(8, 2, 3136, 48, "model"), (24, 16, 128, 49, "shared")]           # both above 2 M scores; rows of 48 and of 49 slots


def _operands(b, h, n, m, kind, seed):
    first, second = (workloads.make_index(kind, b, n, m, s, DEV) for s in (seed, seed + 1))
    g = torch.Generator(device=DEV).manual_seed(seed)
    q, k, v, attn = (torch.randn(b, h, n, w, generator=g, device=DEV) for w in (32, 32, 32, m))
    return first, second, q, k, v, attn


def _check(out, q, k, v, attn, idx):
    assert rel_err(out[0], formula.forward("qk", q.double(), k.double(), idx, chunk=1)) <= TOL[q.dtype]
    assert rel_err(out[1], formula.forward("av", attn.double(), v.double(), idx, chunk=1)) <= TOL[q.dtype]


def _forward(q, k, v, attn, idx):
    from clusten import CLUSTENAVFunction, CLUSTENQKFunction
    return CLUSTENQKFunction.apply(q, k, idx), CLUSTENAVFunction.apply(attn, v, idx)


@pytest.mark.parametrize("size", SIZES, ids=str)
@pytest.mark.parametrize("grad", [False, True])
def test_forward_after_an_untracked_write(lib, size, grad):
    """A write that no version counter sees, as by a replayed graph or another library's kernel."""
    idx, other, q, k, v, attn = _operands(*size, 700)
    q.requires_grad_(grad), attn.requires_grad_(grad)
    _forward(q, k, v, attn, idx)
    version = idx._version
    idx.data.copy_(other)
    assert idx._version == version
    _check(_forward(q, k, v, attn, idx), q.detach(), k, v, attn.detach(), other)


@pytest.mark.parametrize("size", SIZES, ids=str)
def test_replayed_forward_sees_new_indices(lib, size):
    idx, other, q, k, v, attn = _operands(*size, 710)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream), torch.no_grad():
        _forward(q, k, v, attn, idx)                         # the usual warm-up on the static inputs
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph, stream=stream):
        out = _forward(q, k, v, attn, idx)
    idx.copy_(other)
    graph.replay()
    _check(out, q, k, v, attn, other)


@pytest.mark.parametrize("size", SIZES, ids=str)
def test_forward_in_inference_mode(lib, size):
    idx, _, q, k, v, attn = _operands(*size, 720)
    with torch.inference_mode():
        table = idx.clone()
        assert table.is_inference()
        out = _forward(q, k, v, attn, table)
    _check(out, q, k, v, attn, idx)


def test_merge_in_inference_mode(lib):
    from clusten import CLUSTENWFFunction
    b, n_out, n, m, ic, c = 2, 98, 392, 48, 4, 64
    idx = workloads.select_rows(workloads.make_index("model", b, n, m, 730), n_out, 731).to(DEV)
    weights, feat, _ = workloads.merge_operands(b, n_out, n, m, ic, c, torch.float32, 732, DEV)
    with torch.inference_mode():
        out = CLUSTENWFFunction.apply(weights, feat, idx.clone())
    assert rel_err(out, formula.forward("wf", weights.double(), feat.double(), idx)) <= TOL[torch.float32]


def test_replayed_training_step_sees_new_indices(lib):
    """Forward and backward of all three operators, captured after a warm-up; and a call outside the graph before its first replay."""
    from clusten import CLUSTENWFFunction
    b, h, n, m, n_out, ic, c = 2, 2, 392, 48, 98, 4, 64
    idx, other, q, k, v, attn = _operands(b, h, n, m, "model", 740)
    merge, merge_other = (workloads.select_rows(t, n_out, 741) for t in (idx, other))
    weights, feat, grad = workloads.merge_operands(b, n_out, n, m, ic, c, torch.float32, 742, DEV)
    leaf = [t.requires_grad_(True) for t in (q, k, attn, v, weights, feat)]
    ones = [torch.ones(b, h, n, m, device=DEV), torch.ones(b, h, n, 32, device=DEV), grad]

    def step():
        out = (*_forward(q, k, v, attn, idx), CLUSTENWFFunction.apply(weights, feat, merge))
        return [*out, *torch.autograd.grad(out, leaf, ones)]

    def check(got, table, merge_table):
        d = [t.detach().double() for t in (q, k, attn, v, weights, feat)]
        a, dq, dk = formula.forward_backward("qk", d[0], d[1], table, ones[0].double())
        f, da, dv = formula.forward_backward("av", d[2], d[3], table, ones[1].double())
        w, dw, df = formula.forward_backward("wf", d[4], d[5], merge_table, grad.double())
        for i, (x, want) in enumerate(zip(got, (a, f, w, dq, dk, da, dv, dw, df))):
            assert rel_err(x, want) <= TOL[torch.float32], i

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = step()
    check(step(), idx, merge)                               # (nothing that the capture made is taken for built)
    idx.copy_(other), merge.copy_(merge_other)
    torch.cuda.synchronize()
    graph.replay()
    check(out, other, merge_other)


def test_streams_have_buffers_of_their_own(lib):
    from clusten import ops
    idx = workloads.make_index("model", 2, 392, 48, 750, DEV)
    torch.cuda.synchronize()
    found = []
    for stream in (torch.cuda.Stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            found.append((ops.row_order_for(idx), ops.groups_for(idx, 392)))
            assert ops.row_order_for(idx) is found[-1][0] and ops.groups_for(idx, 392) is found[-1][1]
    torch.cuda.synchronize()
    assert found[0][0] is not found[1][0] and found[0][1] is not found[1][1]
    assert torch.equal(found[0][0], found[1][0])
