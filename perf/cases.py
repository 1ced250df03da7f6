"""What a user of the Selective Attention operator has it do, as cases that can be timed and compared.

Every case goes through the public entry points: ``kernels.selective_attention`` (training, any dtype),
``kernels.selective_attention_packed`` (training, on a fused projection output) and ``SelectiveAttentionSlot``
(``attend`` for training a layer, ``begin_cache`` for a prompt, ``extend_cache`` for a further chunk of one,
``step_cache`` for generation).  The sizes are the configurations of the benchmark (T = 16384 training, the 131,072-token
prompt and the decode steps after it, the fp32 case B = 2, H = 4, T = 1024) and ordinary ones around them.
"""

import math
import os
import sys

import torch

PACKAGE = os.path.join(os.getcwd(), "selective-attention-study_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

from selective_attention_b200 import kernels  # noqa: E402
from selective_attention_b200.mixers import SelectiveAttentionSlot  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(kind, name=None, *, batch, heads, seq, dim, dtype="bf16", per_head=False, exempt=1, scale=1.0, skip=False, cached=0,
          steps=0):
    """``seq``: tokens that the call is given (decode: one a step); ``cached``: tokens in the cache before it; ``scale``: of
    q and k, which sets how fast the history term grows; ``skip``: the option that leaves out what has no weight left."""
    c = dict(kind=kind, batch=batch, heads=heads, seq=seq, dim=dim, dtype=dtype, per_head=per_head, exempt=exempt, scale=scale,
             skip=skip, cached=cached, steps=steps)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # the training shape of the benchmark: one layer of a 16-head model at 16K context, head 0 selecting for all
        _case("train", "train-16k", batch=4, heads=16, seq=16384, dim=64),
        # the same layer in the variant where every head selects for itself
        _case("layer", "train-16k-per-head", batch=4, heads=16, seq=16384, dim=64, per_head=True),
        # the same layer with the option that leaves out the tiles without weight, one sequence
        _case("train", "train-16k-live-tiles", batch=1, heads=16, seq=16384, dim=64, skip=True),
        # a 12-head layer at 4K context between its fused projections, as the decoder module calls it
        _case("packed", "layer-4k-packed", batch=2, heads=12, seq=4096, dim=64, scale=0.3),
        # head_dim 128, a length that is no multiple of anything, the first 16 positions exempt
        _case("layer", "train-4097-d128", batch=2, heads=8, seq=4097, dim=128, exempt=16, scale=0.3),
        # the fp32 case that the operator is validated at
        _case("train", "train-1k-fp32", batch=2, heads=4, seq=1024, dim=64, dtype="fp32"),
        # a small fp16 model: short ragged sequences, narrow heads
        _case("layer", "train-1000-fp16-d32", batch=4, heads=8, seq=1000, dim=32, dtype="fp16"),
        # the long prompt: forward, cache and selection totals of 131,072 tokens
        _case("prompt", "prompt-131k", batch=1, heads=16, seq=131072, dim=64),
        # a chat-sized prompt, where latency counts
        _case("prompt", "prompt-300", batch=1, heads=12, seq=300, dim=64, scale=0.3),
        # a further chunk of a long prompt
        _case("extend", "extend-2k-after-30k", batch=1, heads=16, seq=2048, dim=64, cached=30000, scale=0.3),
        # generation after the long prompt: every step streams the cache
        _case("decode", "decode-after-131k", batch=1, heads=16, seq=1, dim=64, cached=131000, steps=4),
        # generation for a small batch of short sequences: latency of a step
        _case("decode", "decode-batch-8", batch=8, heads=12, seq=1, dim=64, cached=1500, steps=8, scale=0.3),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["train", "layer", "packed", "train", "layer", "small", "small", "prompt", "extend", "decode", "decode"])
    scale = rng.choice([1.0, 0.5, 0.3, 0.1])
    exempt = rng.choice([1, 1, 1, 16])
    if kind == "small":       # fp32 and fp16 training, every head_dim, up to 2K context
        dim = rng.choice([16, 32, 64, 128])
        return _case(rng.choice(["train", "layer"]), batch=rng.randint(1, 4), heads=rng.choice([2, 3, 4, 8]),
                     seq=_log(rng, 64, 2048 if dim < 128 else 1024), dim=dim, dtype=rng.choice(["fp32", "fp32", "fp16"]),
                     per_head=rng.random() < 0.2, exempt=exempt, scale=scale)
    dim = rng.choice([64, 64, 64, 128])
    heads = rng.choice([4, 8, 12, 16]) if dim == 64 else rng.choice([2, 4, 8])
    if kind in ("train", "layer", "packed"):
        seq = _log(rng, 128, 16384)
        batch = rng.randint(1, max(1, min(8, 65536 // seq)))
        return _case(kind, batch=batch, heads=heads, seq=seq, dim=dim, per_head=kind == "layer" and rng.random() < 0.4,
                     exempt=exempt, scale=scale, skip=kind == "train" and rng.random() < 0.25)
    per_head = rng.random() < 0.25
    if kind == "prompt":
        seq = _log(rng, 16, 131072 if dim == 64 else 65536)
        if per_head:
            seq = min(seq, 32768)
        return _case(kind, batch=1 if seq > 8192 else rng.randint(1, 2), heads=heads, seq=seq, dim=dim, per_head=per_head,
                     exempt=exempt, scale=scale)
    if kind == "extend":
        return _case(kind, batch=1, heads=heads, seq=_log(rng, 16, 4096), dim=dim, cached=_log(rng, 128, 60000), per_head=per_head,
                     exempt=exempt, scale=scale, skip=rng.random() < 0.3)
    cached = _log(rng, 64, 131000)
    return _case(kind, batch=rng.randint(1, max(1, min(8, 131000 // cached))), heads=heads, seq=1, dim=dim,
                 dtype=rng.choice(["bf16", "bf16", "bf16", "fp16"]), cached=cached, steps=rng.randint(2, 8), per_head=per_head,
                 exempt=exempt, scale=scale, skip=rng.random() < 0.3)


def _normal(gen, shape, scale=1.0, dtype=torch.bfloat16):
    x = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
    return (x * scale if scale != 1.0 else x).to(dtype)


def _slot(c, seq):
    return SelectiveAttentionSlot(c["heads"], seq, exempt=c["exempt"], per_head=c["per_head"])


def _filled_cache(c, gen, capacity):
    """A cache of ``cached`` tokens and the selection that they have received by then.  The keys and values are drawn; the
    selection of a key grows with the queries that came after it, by about what random logits give, and is never negative.
    (A prefill would give the same in kind; this is quick at any length.)"""
    b, h, d, t = c["batch"], c["heads"], c["dim"], c["cached"]
    dtype, groups = DTYPES[c["dtype"]], h if c["per_head"] else 1
    k = torch.zeros(b, h, capacity, d, device="cuda", dtype=dtype)
    v = torch.zeros_like(k)
    k[:, :, :t] = _normal(gen, (b, h, t, d), c["scale"], dtype)
    v[:, :, :t] = _normal(gen, (b, h, t, d), 1.0, dtype)
    later = torch.arange(t - 1, -1, -1, device="cuda", dtype=torch.float32)
    noise = torch.randn(b, groups, t, generator=gen, device="cuda")
    selected = torch.zeros(b, groups, capacity, device="cuda", dtype=torch.float32)
    selected[:, :, :t] = (0.4 * c["scale"] ** 2 * (later + noise * later.sqrt())).clamp_min(0.0)
    selected[:, :, : min(t, c["exempt"])] = 0.0
    cache = {"k": k, "v": v, "len": t, "selected": selected}
    if c["kind"] == "decode" and c["skip"]:
        cache["key_norms"] = kernels.key_norms(k)
    return cache


def prepare(case, seed):
    c = case
    gen = torch.Generator("cuda").manual_seed(seed)
    b, h, t, d = c["batch"], c["heads"], c["seq"], c["dim"]
    dtype = DTYPES[c["dtype"]]
    state = {"case": c}
    if c["kind"] == "packed":
        qkv = torch.empty(b, t, 3, h, d, device="cuda", dtype=dtype)
        for i in range(3):
            qkv[:, :, i] = _normal(gen, (b, t, h, d), c["scale"] if i < 2 else 1.0, dtype)
        return dict(state, qkv=qkv.requires_grad_(True), grad=_normal(gen, (b, t, h * d), 1.0, dtype))
    if c["kind"] in ("train", "layer"):
        q, k = (_normal(gen, (b, h, t, d), c["scale"], dtype).requires_grad_(True) for _ in range(2))
        v = _normal(gen, (b, h, t, d), 1.0, dtype).requires_grad_(True)
        if c["kind"] == "train":          # the operator's own output is fp32, and so is its gradient
            return dict(state, qkv=(q, k, v), grad=_normal(gen, (b, h, t, d), 1.0, torch.float32))
        return dict(state, slot=_slot(c, t), qkv=(q, k, v), grad=_normal(gen, (b, h, t, d), 1.0, dtype))
    if c["kind"] == "prompt":
        qkv = tuple(_normal(gen, (b, h, t, d), s, dtype) for s in (c["scale"], c["scale"], 1.0))
        return dict(state, slot=_slot(c, t + 64), qkv=qkv)
    tokens = t if c["kind"] == "extend" else c["steps"]
    cache = _filled_cache(c, gen, c["cached"] + tokens + 32)
    qkv = tuple(_normal(gen, (b, h, tokens, d), s, dtype) for s in (c["scale"], c["scale"], 1.0))
    if c["kind"] == "decode":
        qkv = [tuple(x[:, :, i:i + 1].contiguous() for x in qkv) for i in range(tokens)]
    return dict(state, slot=_slot(c, cache["k"].shape[2]), cache=cache, prefix=cache["selected"].clone(), qkv=qkv)


def run(state):
    c = state["case"]
    if c["kind"] == "packed":
        y = kernels.selective_attention_packed(state["qkv"], exempt=c["exempt"])
        return [y, *torch.autograd.grad(y, state["qkv"], state["grad"])]
    if c["kind"] == "train":
        q, k, v = state["qkv"]
        y = kernels.selective_attention(q, k, v, exempt=c["exempt"], skip_dead_tiles=c["skip"])
        return [y, *torch.autograd.grad(y, (q, k, v), state["grad"])]
    if c["kind"] == "layer":
        q, k, v = state["qkv"]
        y, _ = state["slot"].attend(q, k, v)
        return [y, *torch.autograd.grad(y, (q, k, v), state["grad"])]
    with torch.no_grad():
        if c["kind"] == "prompt":
            y, cache = state["slot"].begin_cache(*state["qkv"])
            return [y, cache["k"], cache["v"], cache["selected"]]
        # one more continuation of a shared prefix: the cache goes back to the prefix, then on
        cache = state["cache"]
        cache["len"] = c["cached"]
        cache["selected"].copy_(state["prefix"])
        if c["kind"] == "extend":
            y = state["slot"].extend_cache(*state["qkv"], cache, skip_dead_tiles=c["skip"])
            return [y, cache["k"], cache["v"], cache["selected"]]
        ys = [state["slot"].step_cache(q, k, v, cache) for q, k, v in state["qkv"]]
        return [*ys, cache["k"], cache["v"], cache["selected"]]


def _pairs(c):
    """(query, key) pairs of one head, for the selection (every one of them decides the history) and for the attention (with
    ``skip``, those of the keys that can still have weight: a logit has to be 150 binades down, and the history grows by
    about 0.4 scale^2 a query)."""
    t, n = c["seq"], c["cached"]
    every = t * (t + 1) / 2 + t * n
    if not c["skip"]:
        return every, every
    reach = min(t + n, 110.0 / (0.4 * c["scale"] ** 2) + 128)
    return every, min(every, t * reach)


def work(case):
    c = case
    b, h, t, d = c["batch"], c["heads"], c["seq"], c["dim"]
    size, g = {"bf16": 2, "fp16": 2, "fp32": 4}[c["dtype"]], h if c["per_head"] else 1
    rows = b * h
    one = rows * t * d                                          # elements of q (k, v, out, a gradient)
    sel, att = _pairs(c)
    shared = 0 if c["per_head"] else 1                          # a head that selects for itself has its logits already
    forward = b * d * (4 * h * att + 2 * shared * sel)
    if c["kind"] in ("train", "layer", "packed"):
        backward = b * d * (10 * h * att + 6 * shared * att)    # S, dP, dV, dK, dQ; shared: L0 again, and its two gradients
        out = 4 if c["kind"] == "train" else size
        return {"bytes": 6 * one * size + 2 * one * out, "flops": forward + backward}
    if c["kind"] == "prompt":                                   # q, k, v in; y, the cache and its totals out
        return {"bytes": 6 * one * size + 4 * b * g * t, "flops": forward}
    if c["kind"] == "extend":                                   # the cached keys and values, and the new ones
        live = min(c["cached"], att / t)
        return {"bytes": 2 * rows * live * d * size + 6 * one * size + 8 * b * g * (c["cached"] + t), "flops": forward}
    n, steps = c["cached"], c["steps"]
    reach = min(n, 110.0 / (0.4 * c["scale"] ** 2) + 128) if c["skip"] else n
    keys = rows * reach + (b * g * (n - reach) / 2)             # with `skip` a selecting head still reads every key
    return {"bytes": steps * (2 * keys * d * size + 8 * b * g * n), "flops": steps * 4 * d * keys}


def tolerance(case):
    c = case
    if c["kind"] == "decode":                                   # fp32 sums; y comes back in the model's dtype
        return {"rel": 4e-3 if c["dtype"] == "bf16" else 1e-3}
    if c["dtype"] == "bf16":
        # bf16 operands of the products.  A logit that rounds to the other side of zero opens or closes one selection gate,
        # which moves a single term of a gradient by as much as the term is large.
        return {"rel": 1e-2, "max": 0.8}
    return {"rel": {"fp16": 1e-3, "fp32": 1e-5}[c["dtype"]]}
