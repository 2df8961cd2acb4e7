"""Forward with a few query rows: infinite scores and both sides of the line between its two kernels, against fp64 attention;
the same bits from repeats, graph replays and concurrent streams."""

import math

import pytest
import torch

from flashbob_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nq", [1, 2, 4, 8])                 # 8: the sweep kernel, which gives the same
@pytest.mark.parametrize("Nk", [40, 3000])
@pytest.mark.parametrize("entry,width", [(math.inf, 1), (1e30, 1e30), (math.inf, 5)])
def test_an_infinite_score_makes_its_row_nan_and_no_other(Nq, Nk, entry, width):
    """Key 33's score is +inf (an infinite entry, or a product beyond fp32) in the even rows, -inf in the odd ones."""
    gen = torch.Generator().manual_seed(2)
    q, k, v = (torch.randn(2, 3, n, 64, generator=gen) for n in (Nq, Nk, Nk))
    q[..., 0] = torch.tensor([width, -width] * 4)[:Nq]
    k[..., 0] = 0
    k[:, :, 33] = 0
    k[:, :, 33, 0] = entry
    q, k, v = (t.to(torch.bfloat16).cuda() for t in (q, k, v))
    out, _ = ops.attention_forward(q, k, v, is_causal=False, window_size=0, q_offset=0, k_offset=0, scale=None)
    assert out[:, :, 0::2].isnan().all()
    if Nq > 1:
        s = (q[:, :, 1::2].double() @ k.double().transpose(2, 3)) / 8
        s[..., 33] = -math.inf
        # the probabilities of the sweep kernel and every result are rounded to bf16: 2^-8 of a value, or of the sum's scale
        torch.testing.assert_close(out[:, :, 1::2].double(), torch.softmax(s, -1) @ v.double(), rtol=2.0 ** -7, atol=4e-3)


@pytest.mark.parametrize("heads,D,Nk", [
    (32, 128, 200), (33, 128, 200), (64, 64, 300), (65, 64, 300), (128, 32, 600), (129, 32, 600),     # heads x D of a round
    (149, 32, 600), (148, 128, 65), (149, 48, 200),                                                   # ... of two rounds
    (200, 128, 64), (200, 128, 65), (200, 64, 128), (200, 64, 129), (200, 32, 256), (200, 32, 257),   # one round of keys
])
@pytest.mark.parametrize("Nq", [2, 4])
def test_both_sides_of_the_line_between_the_kernels(heads, D, Nk, Nq):
    gen = torch.Generator().manual_seed(6)
    q, k, v = (torch.randn(1, heads, n, D, generator=gen).to(torch.bfloat16).cuda() for n in (Nq, Nk, Nk))
    out, lse = ops.attention_forward(q, k, v, is_causal=True, window_size=0, q_offset=Nk - Nq, k_offset=0, scale=None)
    s = q.double() @ k.double().transpose(2, 3) / math.sqrt(D)
    s = s.masked_fill(torch.ones(Nq, Nk, dtype=torch.bool, device="cuda").triu(Nk - Nq + 1), -math.inf)
    # results are rounded once, by up to 2^-9 of a value (bf16); the kernel for many rows rounds each probability likewise,
    # which moves a result by about 2^-9 sqrt(sum p^2 v^2) < 2^-9 * 0.5: five of that
    torch.testing.assert_close(out.double(), torch.softmax(s, -1) @ v.double(), rtol=2.0 ** -8, atol=5e-3)
    torch.testing.assert_close(lse.double(), torch.logsumexp(s, -1), rtol=2e-5, atol=2e-5)


def _wide(seed, heads=3, Nq=1, Nk=9000, D=64):
    gen = torch.Generator().manual_seed(seed)
    return tuple(torch.randn(2, heads, n, D, generator=gen).to(torch.bfloat16).cuda() for n in (Nq, Nk, Nk))


_FULL = dict(is_causal=False, window_size=0, q_offset=0, k_offset=0, scale=None)


@pytest.mark.parametrize("Nq,D", [(1, 64), (1, 32), (4, 64), (3, 128)])
def test_divided_heads_repeat_bit_for_bit_in_eager_calls_replays_and_streams(Nq, D, monkeypatch):
    """Which CTA of a head finishes last, and adds the parts, differs from run to run; their order does not."""
    monkeypatch.setattr(ops, "_CHECK_STATUS", False)         # reading the status waits, which a capture does not allow
    cases = [_wide(s, Nq=Nq, D=D) for s in range(4)]
    want = [ops.attention_forward(*c, **_FULL) for c in cases]
    same = lambda got, i: torch.equal(got[0], want[i][0]) and torch.equal(got[1], want[i][1])
    for _ in range(50):
        assert same(ops.attention_forward(*cases[0], **_FULL), 0)
    graph = torch.cuda.CUDAGraph()
    static = tuple(t.clone() for t in cases[0])
    with torch.cuda.graph(graph):
        got = ops.attention_forward(*static, **_FULL)
    for i in (0, 1, 2, 3, 0):
        for s, t in zip(static, cases[i]):
            s.copy_(t)
        graph.replay()
        assert same(got, i)
    torch.cuda.synchronize()
    streams, results = [torch.cuda.Stream() for _ in cases], []
    for _ in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                results.append((i, ops.attention_forward(*cases[i], **_FULL)))
    torch.cuda.synchronize()
    assert all(same(got, i) for i, got in results)
