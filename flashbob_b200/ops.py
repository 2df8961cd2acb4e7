"""Tensor-level wrappers of the three C-ABI stages (forward, first backward, second backward).

PyTorch is used only for device memory and streams; all arithmetic happens in libbob_sm100.so, called
through the native host path (csrc/torch_binding.cpp).  After every call a device-side time-out raises:
by default a non-blocking look at the device's host-visible status word (so a time-out of an earlier call
surfaces, at the latest one call late, without synchronising); with BOB_SM100_CHECK_STATUS=1 the call's own
status word is read back after waiting for the stream.
These functions replace the reference's front end and launchers:
`bob.attention.forward` / `first_backward` (reference: src/bob/attention.py:251-289),
`bob.kernels.rectangular.rect_forward` / `rect_first_backward`
(reference: src/bob/kernels/rectangular.py:220-253) and the three second-backward launchers
`square.bob_2pass`, `gqa.bob_gqa`, `rectangular.bob_2pass_rect`
(reference: src/bob/kernels/square.py:383-525, gqa.py:540-718, rectangular.py:628-777).
"""

from __future__ import annotations

import math
import os

import torch

from . import _lib, _native

_CHECK_STATUS = os.environ.get("BOB_SM100_CHECK_STATUS", "0") not in ("", "0")


def _tma_ready(t: torch.Tensor) -> torch.Tensor:
    """Return `t` itself when the kernels can address it in place, else a contiguous copy (what the native
    calls do with their inputs, for callers of the C ABI).

    In-place addressing needs unit stride along the head dim, batch/head/row strides that are
    multiples of 8 elements (16 bytes) and a 16-byte aligned base.
    """
    if t.stride(-1) == 1 and all(s % 8 == 0 for s in t.stride()[:3]) and t.data_ptr() % 16 == 0 \
            and all(s > 0 or n == 1 for s, n in zip(t.stride()[:3], t.shape[:3])):
        return t
    return t.contiguous()


def _set_strides(field, t: torch.Tensor) -> None:
    s = t.stride()
    field[0], field[1], field[2] = s[0], s[1], s[2]


def _geom(q, k, *, is_causal, window_size, q_offset, k_offset, scale) -> _lib.Geom:
    B, Hq, Nq, D = q.shape
    Hkv, Nk = k.shape[1], k.shape[2]
    g = _lib.Geom()
    g.B, g.Hq, g.Hkv, g.Nq, g.Nk, g.D = B, Hq, Hkv, Nq, Nk, D
    g.dtype = _lib.BF16 if q.dtype == torch.bfloat16 else _lib.FP16
    g.is_causal = int(bool(is_causal))
    g.window = int(window_size)
    g.device = q.device.index if q.device.index is not None else torch.cuda.current_device()
    g.q_offset, g.k_offset = int(q_offset), int(k_offset)
    g.scale = float(scale) if scale is not None else 1.0 / math.sqrt(D)
    return g


def _mask(is_causal, window_size, q_offset, k_offset, scale):
    """The mask arguments of the native calls, converted as `_geom` converts them; the C ABI refuses what is out of range."""
    return (bool(is_causal), int(window_size), int(q_offset), int(k_offset), None if scale is None else float(scale), _CHECK_STATUS)


def check_device_status(device=None) -> None:
    """Raise if any libbob_sm100 kernel on `device` gave up on a bounded wait since the last check.
    Non-blocking; call it after a synchronisation point (for instance at the end of a training step)
    to be sure that every kernel launched before it is covered."""
    index = torch.cuda.current_device() if device is None else torch.device(device).index
    st = _lib.load().bob_sm100_last_status(index)
    if st:
        _lib.check(st, f"a libbob_sm100 kernel on cuda:{index}")


def _require_cuda_16bit(*tensors) -> None:
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda:
            raise ValueError("libbob_sm100 kernels take CUDA tensors only")
        if t.dtype not in (torch.float16, torch.bfloat16):
            raise TypeError(f"libbob_sm100 kernels take fp16 or bf16 tensors, got {t.dtype}")


def attention_forward(q, k, v, *, is_causal, window_size, q_offset, k_offset, scale):
    """out [B,Hq,Nq,D] (input dtype) and natural-log lse [B,Hq,Nq] (fp32)."""
    _require_cuda_16bit(q, k, v)
    return _native.load().forward(q, k, v, *_mask(is_causal, window_size, q_offset, k_offset, scale))


def attention_first_backward(q, k, v, out, lse, dO, *, is_causal, window_size, q_offset, k_offset,
                             scale, for_second_order=True):
    """dQ, dK, dV (input dtype, contiguous), delta = rowsum(dO*out) [B,Hq,Nq] (fp32) and, when
    `for_second_order`, pk = softmax(S) K [B,Hq,Nq,D] (fp32) for the second backward (else None)."""
    _require_cuda_16bit(q, k, v, out, dO)
    return _native.load().first_backward(q, k, v, out, lse, dO, *_mask(is_causal, window_size, q_offset, k_offset, scale), for_second_order)


def attention_second_backward(q, k, v, out, lse, delta, pk, dO, dQ, uQ, uK, uV, *, is_causal,
                              window_size, q_offset, k_offset, scale):
    """Qbar, Kbar, Vbar, dObar (input dtype, contiguous).  uQ/uK/uV may be None."""
    _require_cuda_16bit(q, k, v, out, dO, dQ, uQ, uK, uV)
    return _native.load().second_backward(q, k, v, out, lse, delta, pk, dO, dQ, uQ, uK, uV,
                                          *_mask(is_causal, window_size, q_offset, k_offset, scale))
