"""Forward with at most four query rows per head (decode_kernel) against fp64 attention: one CTA per head and
several, ends of a round of keys, every head-dim padding, masks, grouped heads, storage orders."""

import math

import pytest
import torch

from flashbob_b200 import ops

pytestmark = pytest.mark.gpu
BF16, FP16 = torch.bfloat16, torch.float16


@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,D,dtype,mask,order", [
    (1, 2, 2, 1, 1, 64, BF16, {}, "bhnd"),
    (1, 2, 2, 1, 16384, 64, BF16, {}, "bhnd"),                      # 64 splits of a head
    (2, 3, 3, 1, 257, 32, FP16, {}, "bnhd"),                        # half a round
    (2, 3, 3, 1, 513, 32, FP16, {}, "bnhd"),                        # one key past a round: two CTAs, the last with one key
    (2, 3, 3, 1, 257, 64, FP16, {}, "bhnd"),
    (2, 3, 3, 1, 129, 128, BF16, {}, "bnhd"),
    (2, 3, 3, 4, 257, 32, BF16, {}, "bhnd"),                        # (more than one row: rounds half as long)
    (1, 3, 3, 3, 129, 64, BF16, {}, "bnhd"),
    (1, 3, 3, 2, 65, 128, FP16, {}, "bhnd"),
    (1, 2, 2, 1, 5000, 32, BF16, {}, "bhnd"),                       # many parts at head dim 32
    (1, 2, 2, 4, 5000, 32, BF16, {}, "bnhd"),
    (1, 5, 5, 1, 1023, 128, BF16, {}, "bnhd"),
    (3, 200, 200, 1, 129, 64, FP16, {}, "bhnd"),                    # more heads than CTAs wanted: no split
    (2, 4, 4, 4, 2048, 64, BF16, dict(is_causal=True), "bnhd"),     # right-aligned rectangle
    (1, 4, 4, 3, 3001, 128, FP16, dict(is_causal=True, window_size=700), "bhnd"),
    (1, 4, 4, 2, 515, 32, BF16, dict(is_causal=True, window_size=1), "bhnd"),
    (1, 8, 2, 4, 900, 128, BF16, dict(is_causal=True), "bnhd"),     # grouped heads
    (1, 2, 2, 4, 300, 48, BF16, {}, "bhnd"),                        # head dims between the operator's three
    (1, 2, 2, 1, 1300, 112, FP16, {}, "bhnd"),
    (1, 2, 2, 4, 64, 64, BF16, dict(is_causal=True, q_offset=0, k_offset=2), "bhnd"),   # rows without a key
    (1, 2, 2, 4, 4, 64, BF16, dict(is_causal=True), "bhnd"),
])
def test_few_query_rows_match_fp64(B, Hq, Hkv, Nq, Nk, D, dtype, mask, order):
    gen = torch.Generator().manual_seed(7)

    def tensor(H, N):
        t = torch.randn((B, N, H, D) if order == "bnhd" else (B, H, N, D), generator=gen).to(dtype).cuda()
        return t.transpose(1, 2) if order == "bnhd" else t

    q, k, v = tensor(Hq, Nq), tensor(Hkv, Nk), tensor(Hkv, Nk)
    causal, window, k_off = mask.get("is_causal", False), mask.get("window_size", 0), mask.get("k_offset", 0)
    q_off = mask.get("q_offset", Nk - Nq if causal else 0)
    out, lse = ops.attention_forward(q, k, v, is_causal=causal, window_size=window, q_offset=q_off, k_offset=k_off, scale=None)

    kd, vd = (t.double().repeat_interleave(Hq // Hkv, 1) for t in (k, v))
    s = q.double() @ kd.transpose(2, 3) / math.sqrt(D)
    if causal:
        dist = (torch.arange(Nq) + q_off)[:, None] - (torch.arange(Nk) + k_off)[None, :]
        keep = (dist >= 0) & ((dist < window) if window else torch.ones_like(dist, dtype=torch.bool))
        s = s.masked_fill(~keep.cuda(), -math.inf)
    want_lse = torch.logsumexp(s, -1)
    want = torch.nan_to_num((s - want_lse[..., None]).exp(), nan=0.0) @ vd
    # scores, exponents and sums are fp32 (1e-6 each, scores up to about 6 in size); the result is rounded once, by
    # half the spacing of its neighbours: with 8 (bf16) or 11 (fp16) significant bits at most 2^-8 or 2^-11 of a value
    half = 2.0 ** -8 if dtype == BF16 else 2.0 ** -11
    torch.testing.assert_close(out.double(), want, rtol=1.05 * half, atol=2e-5)
    torch.testing.assert_close(lse.double(), want_lse, rtol=2e-5, atol=2e-5)
