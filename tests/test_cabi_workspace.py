"""The forward's workspace: 256 bytes for every geometry, more only for a caller that asked to divide a head's keys."""

import ctypes
import math

import pytest
import torch

from flashbob_b200 import _lib, ops

SPLIT_KEYS = 1


def _geom(B, H, Nq, Nk, D, **mask):
    g = _lib.Geom()
    g.B, g.Hq, g.Hkv, g.Nq, g.Nk, g.D, g.dtype, g.scale = B, H, H, Nq, Nk, D, _lib.BF16, 0.125
    for n, x in mask.items():
        setattr(g, n, x)
    return g


@pytest.mark.parametrize("mask", [{}, dict(is_causal=1, q_offset=100000), dict(is_causal=1, window=3000, q_offset=100000)])
def test_forward_workspace_bytes(mask):
    size = lambda g: _lib.load().bob_sm100_workspace_bytes(_lib.STAGE_FWD, ctypes.byref(g))
    for B, H, D in ((1, 2, 64), (8, 16, 128), (64, 64, 32)):
        for Nq in (1, 2, 4, 5, 8192):
            for Nk in (1, 4096, 100001):
                assert size(_geom(B, H, Nq, Nk, D, **mask)) == 256
    # 2 heads x at most 64 parts of a 64-wide row, its reference and sum, and a counter per head
    assert 256 < size(_geom(1, 2, 1, 100001, 64, flags=SPLIT_KEYS, **mask)) <= 256 + 256 + 2 * 64 * 8 + 2 * 64 * 64 * 4
    assert size(_geom(1, 2, 5, 100001, 64, flags=SPLIT_KEYS)) == 256


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [0, SPLIT_KEYS])
@pytest.mark.parametrize("Nq,D", [(1, 64), (4, 128), (1, 32), (3, 64)])
def test_forward_stays_inside_its_workspace(flags, Nq, D):
    B, H, Nk, guard = 2, 3, 5000, 1 << 22
    gen = torch.Generator().manual_seed(4)
    q, k, v = (torch.randn(B, H, n, D, generator=gen).to(torch.bfloat16).cuda() for n in (Nq, Nk, Nk))
    lib = _lib.load()
    g = ops._geom(q, k, is_causal=False, window_size=0, q_offset=0, k_offset=0, scale=None)
    g.flags = flags
    for field, t in ((g.q_strides, q), (g.k_strides, k), (g.v_strides, v)):
        ops._set_strides(field, t)
    size = lib.bob_sm100_workspace_bytes(_lib.STAGE_FWD, ctypes.byref(g))
    assert (size == 256) == (flags == 0) and size < guard
    ws = torch.full((size + guard,), 0x5a, dtype=torch.uint8, device="cuda")
    out, lse = torch.empty_like(q), torch.empty(B, H, Nq, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = lib.bob_sm100_fwd(ctypes.byref(g), ptr(q), ptr(k), ptr(v), ptr(out), ptr(lse), ptr(ws),
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and lib.bob_sm100_read_status(ptr(ws), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert (ws[size:] == 0x5a).all()
    s = q.double() @ k.double().transpose(2, 3) / math.sqrt(D)
    # fp32 throughout and rounded to bf16 once, 2^-8 of a value; without the flag the kernel for many rows also rounds each
    # probability p to bf16, which moves a result by at most 2^-8 sum(p |v|) <= 2^-8 * 0.8 and in fact by far less: 1e-3
    torch.testing.assert_close(out.double(), torch.softmax(s, -1) @ v.double(), rtol=1.05 * 2.0 ** -8, atol=2e-5 if flags else 1e-3)
    torch.testing.assert_close(lse.double(), torch.logsumexp(s, -1), rtol=2e-5, atol=2e-5)
