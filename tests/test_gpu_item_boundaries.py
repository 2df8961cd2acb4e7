"""What one work item leaves behind for the next in a persistent launch: groups whose last tile lies three or more tiles
back, exchange buffers, items without keys.  Against the oracle on one head, and the same bits on every repeat."""

import pytest
import torch

from flashbob_b200 import ops
from oracle import bob_oracle as O

pytestmark = pytest.mark.gpu


def _check(B, H, Nq, Nk, D, dtype, repeats, second=True, **mask):
    geom = dict(is_causal=mask.get("is_causal", False), window_size=mask.get("window_size", 0),
                q_offset=mask.get("q_offset", 0), k_offset=mask.get("k_offset", 0), scale=None)
    q, k, v, dO, uQ = O.seeded_inputs(11, (B, H, Nq, D), (B, H, Nk, D), dtype, n_extra_q=2)
    uK, uV = O.seeded_inputs(12, (B, H, Nq, D), (B, H, Nk, D), dtype)[1:]
    dq, dk, dv, ddO, duQ, duK, duV = (t.cuda() for t in (q, k, v, dO, uQ, uK, uV))

    def step():
        out, lse = ops.attention_forward(dq, dk, dv, **geom)
        dQ, dK, dV, delta, pk = ops.attention_first_backward(dq, dk, dv, out, lse, ddO, **geom)
        res = dict(out=out, dQ=dQ, dK=dK, dV=dV)
        if second:
            res.update(zip(("Qbar", "Kbar", "Vbar", "dObar"), ops.attention_second_backward(
                dq, dk, dv, out, lse, delta, pk, ddO, dQ, duQ, duK, duV, **geom)))
        return res

    first = step()
    for _ in range(repeats):
        for n, t in step().items():
            assert torch.equal(t, first[n]), n
    one = lambda t: t[-1:, -1:]
    ref = O.bob_closed_form(*(one(t) for t in (q, k, v, dO, uQ, uK, uV)), **geom)
    for n, t in first.items():
        # 16-bit operands and results: 6e-3 (bf16) is what the operator's tests allow everywhere
        assert O.error_metrics(one(t), getattr(ref, n))["l2_rel"] < (6e-3 if dtype == torch.bfloat16 else 1.5e-3), n


@pytest.mark.parametrize("D", [128, 96, 64])
@pytest.mark.parametrize("Nq,Nk,mask", [
    (128, 300, {}),                                                     # three forward tiles per item, every item
    (128, 600, {}),                                                     # five
    (640, 640, dict(is_causal=True)),                                   # 5, 4, 3, 2, 1
    (384, 640, dict(is_causal=True, q_offset=640, window_size=420)),    # a band that leaves the keys: fewer tiles per item
])
def test_items_with_an_odd_number_of_tiles(D, Nq, Nk, mask):
    _check(3, 64, Nq, Nk, D, torch.bfloat16, 20, second=False, **mask)


@pytest.mark.parametrize("D", [128, 80, 64])
def test_items_without_keys_between_items_with_keys(D):
    """Keys start 300 positions after the queries: the first own tiles of every head attend to nothing, and a CTA takes
    such items after others with the row sums of the second backward in its exchange buffer."""
    _check(3, 64, 640, 384, D, torch.bfloat16, 20, is_causal=True, q_offset=0, k_offset=300)
