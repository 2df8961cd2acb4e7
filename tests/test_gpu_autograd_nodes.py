"""What the operator's autograd nodes owe to the rest of PyTorch's autograd: tracing, forward mode, saved-tensor hooks,
checkpointing, batched gradients, release, streams and threads."""

import threading

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


def test_saved_tensor_hooks_see_and_replace_the_saved_tensors():
    leaves, dO, bars = _inputs(0)
    want = _step(causal, leaves, dO, bars)
    packed = []

    def pack(t):
        packed.append(tuple(t.shape))
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        _same(_step(causal, leaves, dO, bars), want)
    # forward: q, k, v, out, lse; first backward kept in the graph: q, k, v, dO, out, lse, dQ, delta, pk
    assert len(packed) == 5 + 9


@pytest.mark.parametrize("reentrant", [False, True])
def test_checkpointed_call_gives_the_same_gradients(reentrant):
    leaves, dO, _ = _inputs(0)
    want = torch.autograd.grad(causal(*leaves), leaves, dO.detach())
    again = [t.detach().requires_grad_(True) for t in leaves]
    out = torch.utils.checkpoint.checkpoint(causal, *again, use_reentrant=reentrant)
    out.backward(dO.detach())
    _same([t.grad for t in again], want)


def test_batched_gradients_are_refused_with_an_error():
    leaves, dO, _ = _inputs(0)
    out = causal(*leaves)
    batch = torch.stack([dO.detach()] * 2)
    for keep in (False, True):
        with pytest.raises(RuntimeError):
            torch.autograd.grad(out, leaves, batch, retain_graph=True, create_graph=keep, is_grads_batched=True)


def test_a_released_graph_is_refused_and_a_retained_one_repeats():
    leaves, dO, bars = _inputs(0)
    out = causal(*leaves)
    a = torch.autograd.grad(out, leaves, dO, retain_graph=True)
    _same(torch.autograd.grad(out, leaves, dO), a)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(out, leaves, dO)
    out = causal(*leaves)
    first = torch.autograd.grad(out, leaves, dO, create_graph=True)
    a = torch.autograd.grad(first, leaves, bars, retain_graph=True)
    _same(torch.autograd.grad(first, leaves, bars), a)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(first, leaves, bars)


def test_an_input_changed_in_place_is_noticed():
    leaves, dO, _ = _inputs(0)
    mid = leaves[0] * 1
    out = causal(mid, *leaves[1:])
    mid.add_(1)
    with pytest.raises(RuntimeError, match="inplace operation"):
        torch.autograd.grad(out, leaves, dO)


@pytest.mark.parametrize("nq", [48, 1])
def test_steps_on_other_streams_and_threads_give_the_same_bits(nq):
    cases = [_inputs(s, nq, 700) for s in range(4)]
    want = [_step(causal, *c) for c in cases]
    torch.cuda.synchronize()
    got, errors = [None] * 4, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    got[i] = _step(causal, *cases[i])
            torch.cuda.synchronize()
        except Exception as e:                  # seen by the main thread below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors
    for g, w in zip(got, want):
        _same(g, w)
