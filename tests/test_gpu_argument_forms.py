"""The operator's native recognition of the usual call against the Python checks, the one statement of what is allowed: for
every form of the arguments both give the same bits or raise the same exception."""

import fractions

import numpy as np
import pytest
import torch

import bob
from flashbob_b200 import _native

pytestmark = pytest.mark.gpu
BF16, FP16 = torch.bfloat16, torch.float16


class _Int(int):
    pass


def _t(*shape, dtype=BF16, device="cuda", seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).to(device)


_SHAPES = dict(square=((1, 4, 40, 64), (1, 4, 40, 64)), tall=((1, 4, 60, 64), (1, 4, 40, 64)), wide=((2, 4, 24, 32), (2, 4, 70, 32)),
               row=((1, 4, 1, 128), (1, 4, 70, 128)), grouped=((1, 8, 40, 64), (1, 2, 40, 64)), grouped_wide=((1, 8, 24, 64), (1, 2, 40, 64)))
_MASKS = [
    {}, dict(is_causal=True), dict(is_causal=np.True_), dict(is_causal=1), dict(is_causal=None),
    dict(is_causal=True, window_size=16), dict(is_causal=True, window_size=40), dict(is_causal=True, window_size=10 ** 6),
    dict(is_causal=True, window_size=2 ** 40), dict(is_causal=True, window_size=2 ** 70), dict(is_causal=True, window_size=-1),
    dict(is_causal=True, window_size=True), dict(is_causal=True, window_size=np.int32(9)), dict(is_causal=True, window_size=_Int(9)),
    dict(is_causal=True, window_size=9.0), dict(is_causal=True, window_size=None), dict(window_size=4),
    dict(is_causal=True, q_offset=30), dict(is_causal=True, q_offset=0), dict(is_causal=True, q_offset=100, k_offset=100),
    dict(is_causal=True, q_offset=0, k_offset=10), dict(is_causal=True, k_offset=7), dict(q_offset=3), dict(k_offset=3), dict(q_offset=-1),
    dict(k_offset=-1), dict(k_offset=None), dict(q_offset=True), dict(q_offset=2.0), dict(is_causal=True, q_offset=np.int64(30)),
    dict(is_causal=True, q_offset=2 ** 41, k_offset=2 ** 41), dict(is_causal=True, q_offset=2 ** 31 + 30, k_offset=2 ** 31, window_size=20),
    dict(scale=0.2), dict(scale=1), dict(scale=0), dict(scale=-0.5), dict(scale=float("nan")), dict(scale=float("inf")), dict(scale=1e300),
    dict(scale=1e-60), dict(scale=True), dict(scale=np.float64(0.2)), dict(scale=np.float32(0.2)), dict(scale=fractions.Fraction(1, 5)),
    dict(scale="0.2"), dict(scale=torch.tensor(0.2)),
]


def _tensors():
    for name, (qs, ks) in _SHAPES.items():
        yield name, (_t(*qs), _t(*ks, seed=1), _t(*ks, seed=2))
    q, k, v = _t(1, 4, 40, 64), _t(1, 4, 40, 64, seed=1), _t(1, 4, 40, 64, seed=2)
    yield "fp16", (q.half(), k.half(), v.half())
    yield "grouped fp16", (_t(1, 8, 40, 64, dtype=FP16), k[:, :2].half(), v[:, :2].half())
    yield "bnhd", tuple(t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v))
    yield "head dim last but one", tuple(t.transpose(2, 3).contiguous().transpose(2, 3) for t in (q, k, v))
    yield "odd row stride", tuple(torch.zeros(1, 4, 40, 67, dtype=BF16, device="cuda")[..., :64].copy_(t) for t in (q, k, v))
    yield "odd base", tuple(torch.zeros(t.numel() + 1, dtype=BF16, device="cuda")[1:].view_as(t).copy_(t) for t in (q, k, v))
    yield "expanded", (q, k[:, :1].expand(-1, 4, -1, -1), v[:, :, :1].expand(-1, -1, 40, -1))
    yield "leaf", (q.clone().requires_grad_(True), k, v)
    yield "parameter", (torch.nn.Parameter(q.clone()), k, v)
    for name, bad in [("fp32", (q.float(), k.float(), v.float())), ("mixed", (q, k.half(), v)), ("mixed v", (q, k, v.float())),
                      ("cpu k", (q, k.cpu(), v)), ("cpu v", (q, k, v.cpu())), ("rank 3", (q[0], k, v)), ("rank 5", (q, k[None], v)),
                      ("head dim 48", (q[..., :48], k[..., :48], v[..., :48])), ("head dims", (q, k[..., :32], v[..., :32])),
                      ("batch", (q, k.expand(2, -1, -1, -1), v.expand(2, -1, -1, -1))), ("v shape", (q, k, v[:, :, :39])),
                      ("heads", (q[:, :3], k[:, :2], v[:, :2])), ("more kv heads", (q[:, :2], k, v)), ("no rows", (q[:, :, :0], k, v)),
                      ("no keys", (q, k[:, :, :0], v[:, :, :0])), ("no heads", (q, k[:, :0], v[:, :0])), ("not a tensor", (q, None, v)),
                      ("list", (q, k, v.tolist())), ("group 64", (_t(1, 64, 8, 32), _t(1, 1, 8, 32), _t(1, 1, 8, 32)))]:
        yield name, bad


def _outcome(args, kw):
    try:
        return bob.sdpa_bob(*args, **kw)
    except Exception as e:
        return e


def test_every_form_of_a_call_gives_what_the_python_checks_give(monkeypatch):
    native = _native.load()
    taken = 0

    def counted(*args, _try=native.try_sdpa):
        nonlocal taken
        out = _try(*args)
        taken += out is not None
        return out

    for name, args in _tensors():
        for kw in _MASKS:
            monkeypatch.setattr(native, "try_sdpa", counted)
            got = _outcome(args, kw)
            monkeypatch.undo()
            monkeypatch.setattr(native, "try_sdpa", lambda *a: None)
            want = _outcome(args, kw)
            monkeypatch.undo()
            assert type(got) is type(want), (name, kw, got, want)
            if isinstance(want, Exception):
                assert str(got) == str(want), (name, kw)
            else:
                assert torch.equal(got, want) and got.requires_grad == want.requires_grad, (name, kw)
    assert taken > 150
