"""Forward with a few query rows: infinite scores, against fp64 attention."""

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
