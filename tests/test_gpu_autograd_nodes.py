"""What the operator's autograd nodes owe to the rest of PyTorch's autograd."""

import pytest
import torch
import torch.autograd.forward_ad as fwAD

import bob

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _inputs(seed, nq=48, nk=48, heads=2, D=64, grad=True):
    g = torch.Generator().manual_seed(seed)
    t = lambda n: torch.randn(1, heads, n, D, generator=g).to(BF16).cuda()
    q, k, v, dO = t(nq), t(nk), t(nk), t(nq)
    bars = (t(nq), t(nk), t(nk))
    return tuple(x.requires_grad_(grad) for x in (q, k, v)), dO.requires_grad_(grad), bars


def _step(op, leaves, dO, bars):
    out = op(*leaves)
    first = torch.autograd.grad(out, leaves, dO, create_graph=True)
    return (out, *first, *torch.autograd.grad(first, (*leaves, dO), bars))


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


causal = lambda q, k, v: bob.sdpa_bob(q, k, v, is_causal=True)


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("nq,nk,kw", [(48, 48, dict(is_causal=True)), (32, 80, dict(is_causal=True)),
                                      (48, 48, dict(is_causal=True, window_size=16)), (48, 70, {}),
                                      (1, 70, dict(is_causal=True, scale=0.2))])
def test_a_traced_call_computes_with_its_inputs(nq, nk, kw):
    op = lambda q, k, v: bob.sdpa_bob(q, k, v, **kw)
    example, leaves = (_inputs(s, nq, nk)[0] for s in (0, 1))
    dO, bars = _inputs(1, nq, nk)[1:]
    with torch.no_grad():
        traced = torch.jit.trace(op, example)
        assert torch.equal(traced(*leaves), op(*leaves))
    traced = torch.jit.trace(op, example)
    for _ in range(3):                          # the first runs profile, the later ones run optimised
        _same(_step(traced, leaves, dO, bars), _step(op, leaves, dO, bars))


def test_a_forward_mode_tangent_of_the_output_gradient_is_refused_where_a_graph_is_kept():
    leaves, dO, _ = _inputs(0)
    out = causal(*leaves)
    with fwAD.dual_level():
        weight = fwAD.make_dual(dO.detach(), torch.ones_like(dO))
        with pytest.raises(NotImplementedError):
            torch.autograd.grad((out * weight).sum(), leaves, create_graph=True)


def test_a_long_chain_of_calls_is_freed_without_recursion():
    q, k, v = (torch.randn(1, 1, 1, 32, device="cuda").to(BF16) for _ in range(3))
    out = q.requires_grad_(True)
    for _ in range(200_000):
        out = bob.sdpa_bob(out, k, v)
    del out                                     # with a stack frame for each call this would overflow the stack
    out = bob.sdpa_bob(q, k, v)
    assert torch.equal(torch.autograd.grad(out.sum(), q)[0], torch.zeros_like(q))      # one key: no dependence on q
