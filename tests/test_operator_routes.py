"""Calls of the autograd operators that must keep their node (CLUSTENQKFunction.apply and its kin), with CPU stand-ins for the kernels."""
import pytest
import torch

from oracle import formula


@pytest.fixture
def stand_ins(lib, monkeypatch):
    from clusten import clusten, ops

    def qk(query, key, nbhd_idx, for_backward=False):
        return formula.qk(query, key, nbhd_idx)
    monkeypatch.setattr(ops, "qk_forward_views", qk)
    monkeypatch.setattr(clusten.CLUSTENQKFunction, "without_grad", staticmethod(qk))
    return clusten.CLUSTENQKFunction


def _args():
    g = torch.Generator().manual_seed(1)
    q, k = torch.randn(1, 2, 8, 32, generator=g), torch.randn(1, 2, 8, 32, generator=g)
    return q, k, torch.randint(8, (1, 8, 4), generator=g)


def test_a_trace_records_the_operator(stand_ins):
    """The kernels behind it are invisible to a trace: without the node it would keep the allocation of the result alone."""
    args = _args()
    with torch.no_grad():
        traced = torch.jit.trace(lambda q, k, i: stand_ins.apply(q, k, i) + 1, args, check_trace=False)
    assert "CLUSTENQKFunction" in str(traced.graph)


@pytest.mark.parametrize("grad", [False, True])
def test_under_compile(stand_ins, grad):
    args = _args()
    args[0].requires_grad_(grad)
    fn = torch.compile(lambda q, k, i: stand_ins.apply(q, k, i) + 1, backend="eager")
    out = fn(*args)
    assert torch.allclose(out, formula.qk(*args) + 1) and out.requires_grad == grad


def test_vmap_is_refused(stand_ins):
    q, k, idx = _args()
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda x: stand_ins.apply(x, k, idx))(q.unsqueeze(0))
