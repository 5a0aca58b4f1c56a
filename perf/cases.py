"""The work that users of this library have it do, as cases that can be timed.

Every case names one public entry point (or, for a model layer, the entry points that the layer calls one
after the other) and the sizes, data type and options of the call:

    path "train"    dilution_attention forward + backward: a training step's attention
    path "layer"    the same inside a model layer: split_heads_rope in front of it, the output handed on in
                    the projection's dtype, gradients back to the fused q/k/v projection
    path "prefill"  dilution_attention_forward(return_aux=True): a prompt's attention and the demand that
                    the cached decode starts from
    path "bid"      kernels_bid.dilution_attention forward + backward: the bid / share ablations
    path "softmax"  softmax_attention_forward: a softmax layer of an alternating model, inference
    path "decode"   dilution_decode_append_step: one token of a dilution layer against its cache
    path "softmax_decode"  softmax_decode_append_step: one token of a softmax layer against its cache

Tensors are (batch, heads, seq, dim).  q, k, v are N(0, 1) (scores of standard deviation 1), upstream
gradients N(0, 0.01^2), as a mean loss over many tokens gives; a cache's demand is what a prefix of that
length has committed on average.
"""

from __future__ import annotations

import importlib
import math

import torch

D = importlib.import_module("dilution-attention_b200")

_DTYPE = {"bf16": torch.bfloat16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp32": 4}
_ROPE_THETA = 10000.0


def listed():
    return [
        # the headline benchmark: one layer's attention of a 16K-context bf16 model, B4 H16
        dict(name="train_16k", path="train", batch=4, heads=16, seq=16384, dim=64, dtype="bf16", precision="bf16"),
        # short-context training: many rows of few tokens
        dict(name="train_1k", path="train", batch=32, heads=12, seq=1024, dim=64, dtype="bf16", precision="bf16"),
        # a rotated layer of a small bf16 model on a batch of ragged length: head split + RoPE, attention,
        # gradients back to c_attn's output
        dict(name="layer_ragged", path="layer", batch=2, heads=8, seq=1777, dim=64, dtype="bf16", precision="bf16"),
        # a 128K-token prompt, one sequence, forward with the decode's starting demand
        dict(name="prefill_128k", path="prefill", batch=1, heads=16, seq=131072, dim=64, dtype="bf16", precision="bf16"),
        # heads of 128, the other common head size of bf16 models
        dict(name="train_d128", path="train", batch=4, heads=8, seq=4096, dim=128, dtype="bf16", precision="bf16"),
        # an fp32 model: the reference runs those with tf32 products
        dict(name="train_fp32", path="train", batch=4, heads=8, seq=4096, dim=64, dtype="fp32", precision="tf32"),
        # the exact fp32 operator at the size of the reference's own parity check
        dict(name="exact_512", path="train", batch=1, heads=4, seq=512, dim=64, dtype="fp32", precision="ieee"),
        # the ablations train at a context of 8192 with 8 heads of 64 in bf16: an element-wise bid ...
        dict(name="bid_sigmoid_8k", path="bid", batch=4, heads=8, seq=8192, dim=64, dtype="bf16", precision="bf16",
             bid="sigmoid", share="inclusive"),
        # ... and a bid that divides by its row's sum
        dict(name="bid_softplus_8k", path="bid", batch=4, heads=8, seq=8192, dim=64, dtype="bf16", precision="bf16",
             bid="softplus", share="inclusive"),
        # a softmax layer of an alternating model reading a batch of prompts
        dict(name="softmax_8k", path="softmax", batch=4, heads=16, seq=8192, dim=64, dtype="bf16", precision="bf16"),
        # serving: 64 sequences of 16K tokens, one new token each
        dict(name="decode_64x16k", path="decode", batch=64, heads=16, seq=16384, dim=64, dtype="bf16"),
        # interactive generation: one sequence, an odd length
        dict(name="decode_one", path="decode", batch=1, heads=16, seq=3001, dim=64, dtype="bf16"),
    ]


# batch * heads * seq^2 of a causal pass that each family may have; the widest matches its listed case
_TRAIN_CELLS = {("bf16", 64): 64 * 16384 ** 2, ("bf16", 128): 32 * 4096 ** 2, ("fp32", 32): 32 * 4096 ** 2,
                ("fp32", 64): 32 * 4096 ** 2, ("fp32", 128): 8 * 4096 ** 2}


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _length(rng, lo, hi):
    """Lengths over their logarithm; a third of them multiples of 128, as training contexts are."""
    n = _log_int(rng, lo, hi)
    return max(lo, n // 128 * 128) if n >= 256 and rng.random() < 0.34 else n


def _rows(rng, most):
    """(batch, heads) with at most `most` rows."""
    heads = rng.choice([h for h in (1, 2, 4, 6, 8, 12, 16) if h <= max(1, most)])
    return _log_int(rng, 1, max(1, min(64, most // heads))), heads


def draw(rng):
    path = rng.choice(("train", "train", "train", "layer", "prefill", "bid", "bid", "softmax", "decode", "decode",
                       "softmax_decode"))
    if path in ("decode", "softmax_decode"):
        dtype = rng.choice(("bf16", "bf16", "bf16", "fp32"))
        dim = rng.choice((64, 64, 64, 128))
        seq = _length(rng, 16, 65536)
        # at most the keys of 64 x 16 rows of 16K, in bytes of cache
        batch, heads = _rows(rng, max(1, min(1024, 2 ** 31 // (seq * dim * _BYTES[dtype]))))
        return dict(path=path, batch=batch, heads=heads, seq=seq, dim=dim, dtype=dtype)
    case = dict(path=path, batch=1, heads=1, seq=1, dim=64, dtype="bf16", precision="bf16")
    cells = 64 * 16384 ** 2
    lo, hi = 64, 16384
    if path == "train":
        case["dtype"], case["dim"], case["precision"] = rng.choice((
            ("bf16", 64, "bf16"), ("bf16", 64, "bf16"), ("bf16", 64, "bf16"), ("bf16", 128, "bf16"), ("fp32", 64, "tf32"),
            ("fp32", 64, "tf32"), ("fp32", 128, "tf32"), ("fp32", 32, "tf32"), ("fp32", 64, "ieee")))
        cells = _TRAIN_CELLS[case["dtype"], case["dim"]]
        hi = 16384 if (case["dtype"], case["dim"]) == ("bf16", 64) else 8192
        if case["precision"] == "ieee":
            cells, hi = 4 * 2048 ** 2, 2048
    elif path == "layer":
        hi = 8192
    elif path == "prefill":
        lo, hi = 128, 131072
    elif path == "bid":
        case["bid"] = rng.choice(("sigmoid", "expshift", "sigshift", "relu", "relu2", "softplus", "softmax"))
        case["share"] = rng.choice(("inclusive", "inclusive", "none")) if case["bid"] != "softmax" else "none"
        cells, hi = 32 * 8192 ** 2, 8192
    case["seq"] = _length(rng, lo, hi)
    most = min(1024, cells // case["seq"] ** 2, (64 * 16384) // case["seq"])
    case["batch"], case["heads"] = _rows(rng, max(1, most))
    return case


def _normal(g, shape, dtype, scale=1.0):
    return torch.empty(shape, device="cuda", dtype=torch.float32).normal_(0.0, scale, generator=g).to(dtype)


def _cache_tensor(g, shape, dtype):
    """A cache is large: filled in the storage type, one batch row at a time."""
    t = torch.empty(shape, device="cuda", dtype=dtype)
    for row in t:
        row.normal_(generator=g)
    return t


class _Rope:
    """The two fields of a model's rotary module that split_heads_rope reads."""

    def __init__(self, dim):
        self.dim, self.theta = dim, _ROPE_THETA


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    b, h, t, d = case["batch"], case["heads"], case["seq"], case["dim"]
    dtype = _DTYPE[case["dtype"]]
    state = dict(case=case)
    if case["path"] in ("decode", "softmax_decode"):
        # a cache that holds t - 1 tokens of at most t (a generation's budget): the call appends the t-th
        state["q1"], state["k1"], state["v1"] = (_normal(g, (b, h, 1, d), dtype) for _ in range(3))
        cache = dict(k=_cache_tensor(g, (b, h, t, d), dtype), v=_cache_tensor(g, (b, h, t, d), dtype), len=t - 1)
        if case["path"] == "decode":
            # position j has collected about sum_{i >= j} 1 / (i + 1) of demand from the queries behind it
            pos = torch.arange(1, t + 1, device="cuda", dtype=torch.float32)
            mean = torch.log(t / pos) + 0.5 / pos
            jitter = torch.empty(b, h, t, device="cuda").uniform_(0.5, 1.5, generator=g)
            cache["committed"] = mean * jitter
        state["cache"] = cache
        return state
    if case["path"] == "layer":
        state["rope"] = _Rope(d)
        state["qkv"] = _normal(g, (b, t, 3 * h * d), dtype).requires_grad_(True)
        state["dout"] = _normal(g, (b, h, t, d), dtype, 1e-2)
        return state
    state["q"], state["k"], state["v"] = (_normal(g, (b, h, t, d), dtype) for _ in range(3))
    if case["path"] in ("train", "bid"):
        for name in "qkv":
            state[name].requires_grad_(True)
        state["dout"] = _normal(g, (b, h, t, d), torch.float32, 1e-2)
    return state


_SHARE = {"inclusive": True, "exclusive": "exclusive", "none": False}


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "decode" or path == "softmax_decode":
        cache = state["cache"]
        cache["len"] = case["seq"] - 1
        step = D.dilution_decode_append_step if path == "decode" else D.softmax_decode_append_step
        y = step(state["q1"], state["k1"], state["v1"], cache)
        return (y, cache["k"], cache["v"]) + ((cache["committed"],) if path == "decode" else ())
    if path == "layer":
        q, k, v = D.split_heads_rope(state["qkv"], case["heads"], state["rope"])
        y = D.dilution_attention(q, k, v, dot_precision=case["precision"]).to(q.dtype)
        (dqkv,) = torch.autograd.grad(y, state["qkv"], state["dout"])
        return y.detach(), dqkv
    q, k, v = state["q"], state["k"], state["v"]
    if path == "prefill":
        out, aux = D.dilution_attention_forward(q, k, v, dot_precision=case["precision"], return_aux=True)
        return out, aux["committed_total"]
    if path == "softmax":
        return D.softmax_attention_forward(q, k, v)
    if path == "bid":
        # the shifted bids divide by the context length, as a model passes it
        out = D.kernels_bid.dilution_attention(q, k, v, dot_precision=case["precision"], bid=case["bid"],
                                               share_cumsum=_SHARE[case["share"]], shift=float(case["seq"]))
    elif case["precision"] == "ieee":
        out = D.dilution_attention_reference(q, k, v)
    else:
        out = D.dilution_attention(q, k, v, dot_precision=case["precision"])
    return (out.detach(), *torch.autograd.grad(out, (q, k, v), state["dout"]))


def work(case):
    """One causal matmul is n t (t + 1) d flops: 7 of them forward + backward (q k^T and share v; then
    q k^T, dout v^T, dv, dq, dk), 2 forward.  Bytes: each input and output once."""
    n, t, d = case["batch"] * case["heads"], case["seq"], case["dim"]
    e = _BYTES[case["dtype"]]
    tensor = n * t * d
    if case["path"] == "decode":       # cache rows, demand read and written, the new token's rows and the output
        return {"bytes": n * t * (2 * d * e + 8) + 6 * n * d * e, "flops": 4 * n * t * d}
    if case["path"] == "softmax_decode":
        return {"bytes": n * t * 2 * d * e + 6 * n * d * e, "flops": 4 * n * t * d}
    causal = n * t * (t + 1) * d
    if case["path"] == "prefill":      # q, k, v; fp32 out; demand
        return {"bytes": tensor * (3 * e + 4) + 4 * n * t, "flops": 2 * causal}
    if case["path"] == "softmax":
        return {"bytes": tensor * 4 * e, "flops": 2 * causal}
    if case["path"] == "layer":        # qkv and dout in, y and dqkv out
        return {"bytes": tensor * 8 * e, "flops": 7 * causal}
    return {"bytes": tensor * (6 * e + 8), "flops": 7 * causal}


def tolerance(case):
    """About four times what each path shows against the same call with fp32 operands and exact fp32 products
    ("ieee"; torch in 64 bits for softmax attention and the decode steps), over lengths from 64 to 16384:
    bf16 operands 1e-3 in the outputs and 3.3e-3 in the gradients, 2-norm, single values up to 4.6e-2;
    tf32 operands 5e-4 and 7e-3; fp32 1e-7.  A bf16 decode step rounds one output row to bf16 (1.7e-3)."""
    if case["path"] in ("decode", "softmax_decode"):
        return {"rel": 7e-3, "max": 2e-2} if case["dtype"] == "bf16" else {"rel": 1e-6, "max": 1e-5}
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3} if case["precision"] == "ieee" else {"rel": 2e-3, "max": 3e-2}
    # relu bids divide the gradient by the mass of their row, which one barely positive score may be all of
    return {"rel": 1.3e-2, "max": 1.0 if case.get("bid") in ("relu", "relu2") else 0.2}
