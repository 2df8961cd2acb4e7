"""`out` with zero strides (one batch element's rows for all) through the C entry of the first backward: no tile of it
can be addressed, its rows are read with plain loads, and the gradients are those of the materialised tensor."""

import ctypes

import pytest
import torch

from flashbob_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,N", [(64, 200), (128, 128), (32, 1)])
def test_first_backward_reads_an_expanded_out(D, N):
    gen = torch.Generator().manual_seed(5)
    B, H = 3, 2
    rand = lambda b: torch.randn(b, H, N, D, generator=gen).to(torch.bfloat16).cuda()
    q, k, v = (rand(1).repeat(B, 1, 1, 1) for _ in range(3))
    dO = rand(B)
    geom = dict(is_causal=True, window_size=0, q_offset=0, k_offset=0, scale=None)
    out, lse = ops.attention_forward(q, k, v, **geom)
    want = ops.attention_first_backward(q, k, v, out, lse, dO, for_second_order=False, **geom)

    lib = _lib.load()
    g = ops._geom(q, k, **geom)
    one = out[:1].contiguous()
    for field, t in ((g.q_strides, q), (g.k_strides, k), (g.v_strides, v), (g.do_strides, dO), (g.out_strides, one.expand(B, -1, -1, -1))):
        ops._set_strides(field, t)
    assert g.out_strides[0] == 0
    dQ, dK, dV = (torch.empty_like(q) for _ in range(3))
    delta = torch.empty_like(lse)
    ws = torch.empty(lib.bob_sm100_workspace_bytes(_lib.STAGE_BWD1, ctypes.byref(g)), dtype=torch.uint8, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = lib.bob_sm100_bwd1(ctypes.byref(g), ptr(q), ptr(k), ptr(v), ptr(one), ptr(lse), ptr(dO), ptr(dQ), ptr(dK), ptr(dV),
                            ptr(delta), None, ptr(ws), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    for a, b in zip((dQ, dK, dV, delta), want):
        # the same sum in the same order: the same bits
        assert torch.equal(a, b)
