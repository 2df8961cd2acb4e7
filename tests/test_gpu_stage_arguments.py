"""Mask arguments of the stage functions: what the C ABI refuses raises, number-likes are converted."""

import math

import numpy as np
import pytest
import torch

from flashbob_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _stages(nq=40, **geom):
    """The results of the three stages, each as a thunk (the later two on the first ones' results at a valid scale)."""
    g = torch.Generator().manual_seed(3)
    q, dO, uQ, k, v, uK, uV = (torch.randn(1, 2, n, 64, generator=g).to(torch.bfloat16).cuda() for n in (nq,) * 3 + (40,) * 4)
    valid = dict(is_causal=True, window_size=8, q_offset=0, k_offset=0, scale=None)
    out, lse = ops.attention_forward(q, k, v, **valid)
    dQ, _, _, delta, pk = ops.attention_first_backward(q, k, v, out, lse, dO, **valid)
    kw = dict(valid, **geom)
    return (lambda: ops.attention_forward(q, k, v, **kw),
            lambda: ops.attention_first_backward(q, k, v, out, lse, dO, **kw),
            lambda: ops.attention_second_backward(q, k, v, out, lse, delta, pk, dO, dQ, uQ, uK, uV, **kw))


@pytest.mark.parametrize("nq", [40, 3])
@pytest.mark.parametrize("bad", [dict(scale=0.0), dict(scale=-1.0), dict(scale=math.nan), dict(scale=math.inf), dict(scale=1e-60),
                                 dict(window_size=-1), dict(q_offset=-1), dict(k_offset=-1), dict(is_causal=False)])
def test_out_of_range_mask_arguments_raise(nq, bad):
    for stage in _stages(nq, **bad):
        with pytest.raises(_lib.BobSm100Error, match="invalid geometry"):
            stage()


@pytest.mark.parametrize("like", [dict(window_size=8.0, scale=np.float32(0.125)), dict(window_size=np.int64(8), q_offset=np.int32(0)),
                                  dict(k_offset=torch.tensor(0), scale=torch.tensor(0.125)), dict(is_causal=1, scale="0.125")])
def test_number_likes_are_converted(like):
    for a, b in zip(_stages(), _stages(**like)):
        for x, y in zip(a(), b()):
            assert torch.equal(x, y)
