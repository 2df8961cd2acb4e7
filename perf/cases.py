"""Performance cases of the attention operator `bob.sdpa_bob`: what users of it run, at their sizes.

A case is one attention layer's work for one step:

  forward  out = sdpa_bob(q, k, v) without gradients: evaluation, prefill, one-token decoding
  train    forward, then the gradients of q, k and v for a given output gradient
  second   forward, first gradients kept in the graph, then their second gradients (for q, k, v and the
           output gradient) along given directions
  hvp      Hessian-vector product of a scalar loss of `out` with respect to q, k and v

`layout` "bnhd" means that q, k and v are views of [B, N, H, D] storage, which is how a model's
projections deliver them; "bhnd" is contiguous [B, H, N, D].  Inputs are N(0, 1).
"""

import math

import torch

import bob

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# matrix products of attending pairs x head dim that each kind cannot do without, in units of one product
# (2 flops per pair and element): forward 2, first backward 5, second backward 12; a Hessian-vector
# product passes through the first backward once more, for the gradient that reaches `out`
_PRODUCTS = {"forward": 2, "train": 7, "second": 19, "hvp": 24}


def _case(name, kind, B, Hq, Hkv, Nq, Nk, D, dtype="bf16", causal=True, window=0, layout="bhnd"):
    c = dict(kind=kind, B=B, Hq=Hq, Hkv=Hkv, Nq=Nq, Nk=Nk, D=D, dtype=dtype, causal=causal, window=window, layout=layout)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one token per sequence against a cache of 4096 keys: a step of text generation
        _case("decode b8 h16 k4096 d64", "forward", 8, 16, 16, 1, 4096, 64),
        # a long grouped-head prompt, read once before generation
        _case("prefill gqa32/8 n8192 d128", "forward", 1, 32, 8, 8192, 8192, 128, layout="bnhd"),
        # evaluating an encoder on short sequences whose length is no multiple of anything
        _case("encode b16 h12 n197 d64 fp16", "forward", 16, 12, 12, 197, 197, 64, dtype="fp16", causal=False, layout="bnhd"),
        # first-order training: a 12-head layer at batch 8, a grouped-head layer, a sliding-window layer
        _case("train b8 h12 n1024 d64", "train", 8, 12, 12, 1024, 1024, 64, layout="bnhd"),
        _case("train b2 gqa32/8 n2048 d128", "train", 2, 32, 8, 2048, 2048, 128, layout="bnhd"),
        _case("train h16 n8192 w1024 d64", "train", 1, 16, 16, 8192, 8192, 64, window=1024),
        # second-order steps: the operator's smallest documented configuration, where only latency and
        # launches count, ...
        _case("second h2 n128 d64", "second", 1, 2, 2, 128, 128, 64),
        # ... a small layer, ...
        _case("second b2 h8 n1024 d64", "second", 2, 8, 8, 1024, 1024, 64),
        # ... a right-aligned rectangle with a window in fp16 (a chunk of queries against its context), ...
        _case("second b4 h16 128x512 w256 d128 fp16", "second", 4, 16, 16, 128, 512, 128, dtype="fp16", window=256),
        # ... bidirectional attention at head dim 32 on a ragged length, ...
        _case("second h8 n2999 d32 full", "second", 1, 8, 8, 2999, 2999, 32, causal=False),
        # ... the Hessian-vector product of the grouped-head benchmark layer, ...
        _case("hvp gqa32/8 n4096 d64", "hvp", 1, 32, 8, 4096, 4096, 64),
        # ... and one batch element of the long-context scaling configuration
        _case("second gqa64/8 n8192 d128", "second", 1, 64, 8, 8192, 8192, 128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("decode", "forward", "train", "second", "second", "hvp"))
    D = rng.choice((32, 64, 64, 128, 128))
    layout = rng.choice(("bhnd", "bnhd"))
    while True:
        B, H = _log_int(rng, 1, 16), rng.choice((2, 4, 8, 12, 16, 24, 32, 64))
        n = _log_int(rng, 128, 16384)
        n -= n % rng.choice((1, 64, 128))               # lengths as they come, and whole tiles
        if kind == "decode":
            c = _case("", "forward", B, H, H, rng.choice((1, 1, 1, 4)), n, D, dtype=rng.choice(("bf16", "fp16")), layout=layout)
        else:
            mask = rng.choice(("grouped", "grouped", "causal", "causal", "full", "window", "rectangle"))
            if mask == "grouped":
                G = rng.choice([g for g in (2, 3, 4, 8) if H % g == 0])
                c = _case("", kind, B, H, H // G, n, n, D, layout=layout)
            else:
                nq = n if mask != "rectangle" else max(128, n // rng.choice((2, 4, 8)))
                window = _log_int(rng, 128, 2048) if mask in ("window", "rectangle") and n > 256 else 0
                c = _case("", kind, B, H, H, nq, n, D, dtype=rng.choice(("bf16", "bf16", "fp16")), causal=mask != "full",
                          window=window if window < n else 0, layout=layout)
        w = work(c)
        if w["flops"] <= 5e12 and w["bytes"] <= 2e9:    # no more than about half of the largest listed case
            return c


def prepare(case, seed):
    B, Hq, Hkv, Nq, Nk, D = (case[x] for x in ("B", "Hq", "Hkv", "Nq", "Nk", "D"))
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def tensor(H, N, grad=False):
        shape = (B, N, H, D) if case["layout"] == "bnhd" else (B, H, N, D)
        t = torch.randn(shape, dtype=_DTYPES[case["dtype"]], device="cuda", generator=gen)
        if case["layout"] == "bnhd":
            t = t.transpose(1, 2)
        return t.requires_grad_(grad)

    grad = case["kind"] != "forward"
    state = dict(kind=case["kind"], kw=dict(is_causal=case["causal"], window_size=case["window"]),
                 q=tensor(Hq, Nq, grad), k=tensor(Hkv, Nk, grad), v=tensor(Hkv, Nk, grad))
    if case["kind"] in ("train", "second"):
        state["dO"] = tensor(Hq, Nq, case["kind"] == "second")
    if case["kind"] in ("second", "hvp"):
        state["directions"] = (tensor(Hq, Nq), tensor(Hkv, Nk), tensor(Hkv, Nk))
    return state


def run(state):
    kind, leaves = state["kind"], (state["q"], state["k"], state["v"])
    if kind == "forward":
        with torch.no_grad():
            return bob.sdpa_bob(*leaves, **state["kw"])
    out = bob.sdpa_bob(*leaves, **state["kw"])
    if kind == "train":
        return out.detach(), *torch.autograd.grad(out, leaves, state["dO"])
    if kind == "second":
        first = torch.autograd.grad(out, leaves, state["dO"], create_graph=True)
        second = torch.autograd.grad(first, leaves + (state["dO"],), state["directions"])
        return (out.detach(), *(t.detach() for t in first), *second)
    loss = out.float().square().sum()
    first = torch.autograd.grad(loss, leaves, create_graph=True)
    return (loss.detach(), *(t.detach() for t in first), *torch.autograd.grad(first, leaves, state["directions"]))


def _pairs(case):
    """Attending (query, key) pairs of one head; queries are right-aligned with the keys."""
    Nq, Nk, window = case["Nq"], case["Nk"], case["window"]
    if not case["causal"]:
        return Nq * Nk
    shift = Nk - Nq if Nk > Nq else 0
    return sum(min(i + shift + 1, window or i + shift + 1, Nk) for i in range(Nq))


def work(case):
    q_side, k_side = case["B"] * case["Hq"] * case["Nq"] * case["D"], case["B"] * case["Hkv"] * case["Nk"] * case["D"]
    # tensors read and written, of the query's size and of the keys' size
    n_q, n_k = {"forward": (2, 2), "train": (4, 4), "second": (7, 8), "hvp": (5, 8)}[case["kind"]]
    return {"bytes": 2 * (n_q * q_side + n_k * k_side),
            "flops": 2 * _PRODUCTS[case["kind"]] * _pairs(case) * case["B"] * case["Hq"] * case["D"]}


def tolerance(case):
    # the derived operands of the matrix products and the results are rounded to the input type: half an ulp is
    # 2^-9 (bf16) or 2^-12 (fp16), and a second gradient is a sum of differences of such terms
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3, "max": 0.1}
