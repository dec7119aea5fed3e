"""The attention calls that this package is measured on.

``listed()`` names twelve calls from the smallest to the largest; ``draw`` gives further calls from
the same ranges.  ``prepare`` makes what a program holds before the call, ``run`` makes the call
through the public entry points, ``work`` counts the bytes and operations the call cannot do
without, ``tolerance`` says how far two correct implementations may differ.

A case is a dict:

``entry``   the public entry point
            ``mask``   ``ops.mha_fwd_with_mask``
            ``lse``    ``ops.mha_fwd_with_mask_lse``
            ``rule``   ``ops.mha_fwd_rule_mask`` (the mask as a rule, no mask tensor)
            ``built``  ``masks.rule_mask`` and then ``ops.mha_fwd_with_mask`` on the mask it wrote
            ``host``   ``mha_fwd_with_mask_from_host`` (all operands in pinned host memory)
``B H Hk Sq Sk d dtype``   the shape; q is (B, H, Sq, d), k and v are (B, Hk, Sk, d)
``kind``    what the mask hides, see ``_mask``; for ``rule`` and ``built`` one of causal,
            causal_window, padding, causal_padding
"""
from __future__ import annotations

import math

import torch

from custom_ops_b200 import masks, mha_fwd_with_mask_from_host, ops

WINDOW = 512
RULE_KINDS = ("causal", "causal_window", "padding", "causal_padding")
MASK_KINDS = ("random10", "bias", "item_sparse", "padding_random") + RULE_KINDS

# No drawn case costs more than the largest listed one: dense operations, bytes of K and V, of the mask.
MAX_FLOPS, MAX_KV_BYTES, MAX_MASK_BYTES = 1.1e12, 2.7e8, 1.35e8


def _case(name, entry, B, H, Hk, Sq, Sk, d, dtype, kind):
    c = dict(entry=entry, B=B, H=H, Hk=Hk, Sq=Sq, Sk=Sk, d=d, dtype=dtype, kind=kind)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # The smallest call: a short sequence with few heads, where the launch and the host path count.
        _case("small", "mask", 2, 4, 4, 256, 256, 64, "bf16", "random10"),
        # One token per sequence against a padded key/value cache: the step of a decoding loop.
        _case("decode", "mask", 8, 16, 4, 1, 4096, 128, "bf16", "padding"),
        # A batch of prompts of unequal, odd length: the padded causal mask is built, then used.
        _case("padded_prompts", "built", 8, 16, 16, 777, 777, 64, "bf16", "causal_padding"),
        # The headline shape: a dense prefill under an unstructured 0 / -inf mask.
        _case("standard", "mask", 4, 16, 16, 2048, 2048, 128, "bf16", "random10"),
        # Finite relative-position biases with dropped keys; fp16, the smaller head, and the LSE as
        # a caller wants it that merges key ranges or computes a backward pass.
        _case("bias_lse_d64", "lse", 4, 16, 16, 2048, 2048, 64, "fp16", "bias"),
        # Grouped-query prefill under a causal sliding window, given as a tensor ...
        _case("gqa_window", "mask", 4, 16, 4, 2048, 2048, 128, "bf16", "causal_window"),
        # ... and the same call with the window given as a rule.
        _case("window_rule", "rule", 4, 16, 4, 2048, 2048, 128, "bf16", "causal_window"),
        # A chunk of a long prompt against the keys cached so far, plus its own.
        _case("chunk_rule", "rule", 1, 32, 8, 512, 4608, 128, "bf16", "causal"),
        # Few query rows over a very long, padded context: the keys have to be split over the GPU.
        _case("splitkv_long", "mask", 1, 16, 16, 128, 32768, 128, "bf16", "padding_random"),
        # Ranking with items of eight tokens; neither length is a multiple of anything.
        _case("ragged_items", "mask", 4, 16, 4, 1000, 4099, 128, "fp16", "item_sparse"),
        # The largest call: the prefill of a long prompt under a causal mask.
        _case("long_causal", "mask", 1, 32, 8, 8192, 8192, 128, "bf16", "causal"),
        # The headline shape with all operands in host memory.
        _case("from_host", "host", 4, 16, 16, 2048, 2048, 128, "bf16", "random10"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    while True:
        family = rng.choices(("prefill", "chunk", "decode", "long", "host"), (9, 3, 3, 3, 1))[0]
        H = rng.choice((4, 8, 12, 16, 24, 32))
        Hk = H // rng.choice([g for g in (1, 1, 2, 4, 8) if H % g == 0])
        d = rng.choice((64, 128, 128))
        dtype = rng.choice(("bf16", "bf16", "fp16"))
        B = _log_int(rng, 1, 16)
        if family == "prefill":
            entry = rng.choices(("mask", "lse", "rule", "built"), (5, 2, 2, 1))[0]
            Sq = Sk = _log_int(rng, 96, 8192)
            if rng.random() < 0.3:                                  # keys of another length than the queries
                Sk = _log_int(rng, 96, 8192)
        elif family == "chunk":
            entry = rng.choice(("mask", "rule", "rule"))
            Sq = _log_int(rng, 64, 1024)
            Sk = Sq + _log_int(rng, 256, 16384)
        elif family == "decode":
            entry = rng.choice(("mask", "mask", "lse", "rule"))
            Sq = rng.choice((1, 1, 1, 2, 4, 7))
            Sk = _log_int(rng, 256, 16384)
            B = _log_int(rng, 1, 32)
        elif family == "long":
            entry = rng.choice(("mask", "mask", "lse"))
            B, Sq, Sk = rng.choice((1, 1, 2)), _log_int(rng, 8, 256), _log_int(rng, 8192, 32768)
        else:
            entry, B, Sq, Sk = "host", _log_int(rng, 2, 8), _log_int(rng, 256, 2048), _log_int(rng, 256, 2048)
        if rng.random() < 0.5:                                      # half of the lengths are round, half are not
            Sq, Sk = (-(-x // 64) * 64 if x > 32 else x for x in (Sq, Sk))
        if entry in ("rule", "built") or family in ("chunk", "decode"):
            kind = rng.choice(RULE_KINDS if family != "decode" else ("padding", "causal_padding"))
        else:
            kind = rng.choice(MASK_KINDS)
        if Sk < Sq and "causal" in kind:
            continue
        c = _case(None, entry, B, H, Hk, Sq, Sk, d, dtype, kind)
        if (_dense_flops(c) <= MAX_FLOPS and 4 * B * Hk * Sk * d <= MAX_KV_BYTES and
                2 * B * Sq * Sk <= MAX_MASK_BYTES and (entry != "host" or _dense_flops(c) <= 1.4e11)):
            return c


def _dense_flops(c):
    return 4.0 * c["B"] * c["H"] * c["Sq"] * c["Sk"] * c["d"]


def _valid_lens(c):
    """Lengths of a padded batch, spread evenly over (Sk / 2, Sk]: the same for every seed, so that
    the work of a case is known."""
    B, Sk = c["B"], c["Sk"]
    return [Sk - (i * (Sk // 2)) // B for i in range(B)] if B > 1 else [max(1, (Sk * 9) // 10)]


def _mask(c, gen):
    """The additive mask (B, 1, Sq, Sk): 0 visible, -inf hidden, finite where the kind says so."""
    B, Sq, Sk, kind = c["B"], c["Sq"], c["Sk"], c["kind"]
    i = torch.arange(Sq, device="cuda").view(1, Sq, 1) + (Sk - Sq)
    j = torch.arange(Sk, device="cuda").view(1, 1, Sk)
    dtype = torch.bfloat16 if c["dtype"] == "bf16" else torch.float16
    m = torch.zeros(B, 1, Sq, Sk, dtype=dtype, device="cuda")
    for b in range(B):
        hide = torch.zeros(1, Sq, Sk, dtype=torch.bool, device="cuda")
        if kind in ("random10", "bias", "padding_random"):         # every tenth key, never the first
            hide = torch.rand(1, Sq, Sk, device="cuda", generator=gen) < 0.1
            hide[..., 0] = False
        if kind == "item_sparse":                                  # items of eight keys, never the first eight items
            items = torch.rand(1, Sq, -(-Sk // 8), device="cuda", generator=gen) < 0.1
            hide = items.repeat_interleave(8, dim=-1)[..., :Sk].clone()
            hide[..., :64] = False
        if "causal" in kind:
            hide |= j > i
        if kind == "causal_window":
            hide |= j <= i - WINDOW
        if kind == "padding_random":
            hide[..., max(1, (Sk * 9) // 10):] = True
        if kind in ("padding", "causal_padding"):
            hide |= j >= _valid_lens(c)[b]
        if kind == "bias":
            m[b, 0] = torch.randn(Sq, Sk, device="cuda", generator=gen) * 0.3
        m[b].masked_fill_(hide, float("-inf"))
    return m


def prepare(case, seed):
    c = dict(case)
    ops.ensure_loaded("fa")
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.bfloat16 if c["dtype"] == "bf16" else torch.float16
    sigma = 0.5 if c["kind"] == "item_sparse" else 1.0

    def normal(heads, rows):
        return torch.randn(c["B"], heads, rows, c["d"], device="cuda", dtype=dtype, generator=gen) * sigma

    s = dict(entry=c["entry"], q=normal(c["H"], c["Sq"]), k=normal(c["Hk"], c["Sk"]), v=normal(c["Hk"], c["Sk"]))
    if c["entry"] in ("rule", "built"):
        s["causal"] = "causal" in c["kind"]
        s["window"] = WINDOW if c["kind"] == "causal_window" else 0
        s["lens"] = (torch.tensor(_valid_lens(c), dtype=torch.int32, device="cuda")
                     if "padding" in c["kind"] else None)
        s["shape"], s["dtype"] = (c["B"], c["Sq"], c["Sk"]), dtype
    else:
        s["mask"] = _mask(c, gen)
    if c["entry"] == "host":
        for name in ("q", "k", "v", "mask"):
            s[name] = s[name].cpu().pin_memory()
    return s


def run(state):
    s, entry = state, state["entry"]
    if entry == "mask":
        return ops.mha_fwd_with_mask(s["q"], s["k"], s["v"], s["mask"])
    if entry == "lse":
        return ops.mha_fwd_with_mask_lse(s["q"], s["k"], s["v"], s["mask"])
    if entry == "rule":
        return ops.mha_fwd_rule_mask(s["q"], s["k"], s["v"], causal=s["causal"], window=s["window"],
                                     valid_lens=s["lens"])
    if entry == "built":
        mask = masks.rule_mask(*s["shape"], dtype=s["dtype"], causal=s["causal"], window=s["window"],
                               valid_lens=s["lens"])
        return ops.mha_fwd_with_mask(s["q"], s["k"], s["v"], mask)
    return mha_fwd_with_mask_from_host(s["q"], s["k"], s["v"], s["mask"])


def _visible(c):
    """(visible (query, key) pairs, keys that any query of a batch element sees), summed over the
    batch.  Keys hidden by chance count as visible: there are some in every neighbourhood."""
    Sq, Sk, kind = c["Sq"], c["Sk"], c["kind"]
    pairs = keys = 0
    for b in range(c["B"]):
        limit = Sk
        if kind in ("padding", "causal_padding"):
            limit = _valid_lens(c)[b]
        if kind == "padding_random":
            limit = max(1, (Sk * 9) // 10)
        if "causal" in kind:
            hi = [min(limit - 1, i + Sk - Sq) for i in range(Sq)]
            lo = [max(-1, i + Sk - Sq - WINDOW) if kind == "causal_window" else -1 for i in range(Sq)]
            pairs += sum(max(0, h - l) for h, l in zip(hi, lo))
            keys += max(hi) + 1 - (min(lo) + 1)
        else:
            pairs += Sq * limit
            keys += limit
    return pairs, keys


def work(case):
    c = case
    pairs, keys = _visible(c)
    nbytes = 2.0 * (2 * c["B"] * c["H"] * c["Sq"] * c["d"] + 2 * c["Hk"] * keys * c["d"])
    if c["entry"] not in ("rule", "built"):
        nbytes += 2.0 * c["B"] * c["Sq"] * c["Sk"]
    if c["entry"] == "lse":
        nbytes += 4.0 * c["B"] * c["H"] * c["Sq"]
    return {"bytes": nbytes, "flops": 4.0 * c["H"] * c["d"] * pairs}


def tolerance(case):
    # P and the output are rounded to the input type (2^-9 or 2^-12 relative to nearest, each);
    # sums, maxima and the LSE are fp32.
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}


def exact(case, seed):
    """What ``run`` returns for these inputs, in 64 bits: one head at a time, so that the scores of
    the largest call fit the card several times over."""
    c = dict(case)
    s = prepare(c, seed)
    mask = (s["mask"] if "mask" in s else _mask(c, None)).cuda()
    q, k, v = (s[n].cuda() for n in ("q", "k", "v"))
    out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    lse = torch.empty(q.shape[:3], dtype=torch.float64, device="cuda")
    for b in range(c["B"]):
        m = mask[b, 0].double()
        for h in range(c["H"]):
            kv = h // (c["H"] // c["Hk"])
            x = torch.addmm(m, q[b, h].double(), k[b, kv].double().T, alpha=1.0 / math.sqrt(c["d"]))
            lse[b, h] = torch.logsumexp(x, dim=-1)
            # a row that sees no key gives 0
            p = x.sub_(lse[b, h].clamp_min(-1e300).unsqueeze(-1)).exp_()
            out[b, h] = p @ v[b, kv].double()
    if c["entry"] == "lse":
        return out, lse
    return out.cpu() if c["entry"] == "host" else out
