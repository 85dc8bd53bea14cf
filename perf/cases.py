"""The work a user of this package has it do, as measurable cases.

Four kinds, all through the public entry points:

* ``decode``  one decode step over a stack of layers: ``qkv_matmul_hqe_2`` on every layer's tiered cache, issued from
              Python as a model issues it.  ``layers`` caches of their own, so that a step reads more than the L2
              holds wherever the model's own step does.
* ``layer``   the same with what surrounds it in an attention layer: the new K / V row is appended to the residual
              window before the call and the head-summed probability row goes into the importance ring after it.
* ``flush``   the residual window moves into the tiers: importance of every token from the ring, block ranking,
              ``KV_cache_hqe_2``.  ``history`` = 0 is the flush that ends a prefill (everything is quantised from
              fp16), otherwise one of the small flushes that follow every 32 decoded tokens.
* ``codec``   quantise + pack of K (along tokens) and V (along channels) and the dequantisation of both.

Shapes are those of ``hqekv_b200.configs`` and ``hqekv_b200.sweep`` (8 kv heads x 128 channels, four query heads per kv
head, Llama-3.1-8B / Qwen3-8B), data is N(0, 1) in fp16 with a few x10 outlier channels in K.
"""
import math

import torch

from hqekv_b200.configs import CacheConfig, tier_counts
from hqekv_b200.model.public_func import get_block_token_idx, last_attn_weights
from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
from hqekv_b200.quant.hqe_matmul import qkv_matmul_hqe_2
from hqekv_b200.quant.pack_unpack import (uniform_group_dequantize_unpack_last_dim,
                                          uniform_group_quantize_pack_last_dim)

D = 128
RING_ROWS = 20          # decode steps the importance ring remembers
UNIFORM = "uniform_group"
CODEBOOK = "high_uniform_group_low_normal_group"   # 1-bit tier in the Gaussian codebook, 64 tokens kept in fp16

# shares of the surviving tokens in the 8-, 4-, 2- and 1-bit tiers, and the strategy they are used with
MIXES = {
    "20/40/40": ((0.20, 0.40, 0.40, 0.0), UNIFORM),
    "25/50/25": ((0.25, 0.50, 0.25, 0.0), UNIFORM),
    "10/25/65": ((0.10, 0.25, 0.65, 0.0), UNIFORM),
    "all4": ((0.0, 1.0, 0.0, 0.0), UNIFORM),
    "all2": ((0.0, 0.0, 1.0, 0.0), UNIFORM),
    "all8": ((1.0, 0.0, 0.0, 0.0), UNIFORM),
    "thirds": ((0.0, 1 / 3, 1 / 3, 1 / 3), CODEBOOK),
}


# ------------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------------
def _attn(kind, name, batch, flushed, residual, mix, evict, group, layers, kv=8, rep=4):
    return {"name": name, "kind": kind, "batch": batch, "kv_heads": kv, "rep": rep, "flushed": flushed,
            "residual": residual, "mix": mix, "evict": evict, "group": group, "layers": layers}


def _flush(name, batch, history, window, keep, mix, evict, group, times_range, kv=8):
    return {"name": name, "kind": "flush", "batch": batch, "kv_heads": kv, "history": history, "window": window,
            "keep": keep, "mix": mix, "evict": evict, "group": group, "times_range": times_range}


def _codec(name, batch, tokens, bit, group, kv=8):
    return {"name": name, "kind": "codec", "batch": batch, "kv_heads": kv, "tokens": tokens, "bit": bit, "group": group}


def listed():
    return [
        # one layer at 4k context: the smallest call, bound by launches and the host (configuration 0)
        _attn("decode", "decode-1layer-4k", 1, 3968, 128, "25/50/25", 0.10, 32, 1),
        # batch-1 decode of an 8B model at 32k context, half of its 32 layers (configuration 1)
        _attn("decode", "decode-b1-32k", 1, 32640, 128, "20/40/40", 0.10, 32, 16),
        # batched serving, groups of 64, a residual window in the middle of filling up (configuration 2)
        _attn("decode", "decode-b8-16k-g64", 8, 16256, 109, "25/50/25", 0.0, 64, 6),
        # long context at batch 4: the largest decode (configuration 3)
        _attn("decode", "decode-b4-128k", 4, 130816, 256, "10/25/65", 0.30, 32, 2),
        # many short sequences, one uniform width and groups of 128 (a point of the kernel sweep)
        _attn("decode", "decode-b32-4k-all4-g128", 32, 3968, 131, "all4", 0.0, 128, 6),
        # a decode layer of the model harness: append, attend over fp16 + 4/2/1-bit tiers, importance row
        _attn("layer", "layer-b1-32k-codebook", 1, 32640, 45, "thirds", 0.25, 32, 8),
        # the flush after 32 decoded tokens, shares of the model harness
        _flush("flush-32-into-24k", 1, 24480, 32, 13, "thirds", 0.0, 32, True),
        # the same for a batch of eight in a cache of bounded length: every flush evicts a block
        _flush("flush-32-into-16k-b8", 8, 16256, 32, 0, "25/50/25", 0.002, 32, True),
        # end of a 32k prefill: everything is ranked, a tenth evicted, the rest quantised
        _flush("flush-prefill-32k", 1, 0, 32640, 128, "20/40/40", 0.10, 32, False),
        # end of a prefill of eight sequences of odd length
        _flush("flush-prefill-b8-5k", 8, 0, 5152, 21, "25/50/25", 0.0, 32, True),
        # the codec alone over a long prompt
        _codec("codec-128k-4bit", 1, 131072, 4, 32),
        # and over short ragged ones, groups of 64
        _codec("codec-b2-3k-2bit-g64", 2, 3136, 2, 64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "layer", "flush", "codec"))
    kv = rng.choice((8, 8, 8, 4, 2, 1))           # all heads of a layer, or a GPU's share of them
    group = rng.choice((32, 32, 64, 128))
    if kind in ("decode", "layer"):
        ctx = _log(rng, 1000, 130000)
        mix = rng.choice(tuple(MIXES))
        if mix == "thirds":
            group = 32
        case = {"kind": kind, "batch": max(1, min(64, round(_log(rng, 1, 64)))), "kv_heads": kv,
                "rep": rng.choice((4, 4, 4, 8, 2)), "flushed": max(8, int(ctx) // group) * group,
                "residual": rng.randint(1, 190), "mix": mix, "evict": rng.choice((0.0, 0.1, 0.3)), "group": group, "layers": 1}
        while case["batch"] > 1 and work(case)["bytes"] > 4.5e8:
            case["batch"] //= 2
        case["layers"] = max(1, min(12, int(9e8 / work(case)["bytes"])))
        return case
    if kind == "flush":
        ctx = _log(rng, 1000, 60000)
        batch = max(1, min(8, round(_log(rng, 1, 8)), int(100000 * 8 / kv / ctx)))
        mix = rng.choice(("20/40/40", "25/50/25", "10/25/65", "thirds"))
        group = 32 if mix == "thirds" else rng.choice((32, 32, 64))
        n = max(16, int(ctx) // group) * group
        prefill = rng.random() < 0.4
        return {"kind": kind, "batch": batch, "kv_heads": kv, "history": 0 if prefill else n,
                "window": n if prefill else group, "keep": rng.randint(0, group - 1), "mix": mix,
                "evict": rng.choice((0.1, 0.25)) if prefill else rng.choice((0.0, 0.002)), "group": group,
                "times_range": rng.random() < 0.5}
    tokens = _log(rng, 500, 100000)
    batch = max(1, min(8, round(_log(rng, 1, 8)), int(100000 * 8 / kv / tokens)))
    return {"kind": kind, "batch": batch, "kv_heads": kv, "tokens": max(4, int(tokens) // group) * group,
            "bit": rng.choice((8, 4, 2)), "group": group}


def _config(case, flushed, residual, evict):
    """The package's description of a cache with ``flushed`` tokens quantised in one go."""
    shares, strategy = MIXES[case["mix"]]
    return CacheConfig("", case["batch"], case["kv_heads"] * case.get("rep", 4), case["kv_heads"], D, flushed + residual,
                       residual, shares, evict, case["group"], True, 1, 64 if strategy == CODEBOOK else 0, strategy)


def _share_evicted(case):
    """Of all tokens ranked in a flush; a small flush that evicts makes room for at least one block."""
    if case["history"] and case["evict"]:
        return max(case["evict"], case["group"] / (case["history"] + case["window"]))
    return case["evict"]


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _kv(gen, batch, heads, tokens):
    """K and V [batch, heads, tokens, 128] fp16; four of a head's K channels are outliers."""
    k = torch.randn(batch, heads, tokens, D, generator=gen, device="cuda", dtype=torch.float16)
    v = torch.randn(batch, heads, tokens, D, generator=gen, device="cuda", dtype=torch.float16)
    gain = torch.ones(1, heads, 1, D, device="cuda", dtype=torch.float16)
    channels = torch.rand(heads, D, generator=gen, device="cuda").argsort(-1)[:, :4]
    gain.view(heads, D).scatter_(1, channels, 10.0)
    return k.mul_(gain), v


def _levels(gen, counts, group):
    """How much every block of ``group`` tokens matters, 0 the most: as many blocks of each level as ``counts`` has
    tokens, scattered over the text."""
    blocks = torch.tensor([n // group for n in counts], device="cuda")
    levels = torch.arange(len(counts), device="cuda").repeat_interleave(blocks)
    return levels[torch.randperm(levels.numel(), generator=gen, device="cuda")]


def _later_levels(gen, levels, counts, group):
    """The levels a few steps later: one block more, which matters the most, every twentieth block of the old order
    has traded places with another one, and ``counts`` says how many blocks each level now takes.  (Which blocks is a
    matter of the seed, how many change their tier is not.)"""
    order = torch.argsort(levels.float() + 0.5 * torch.rand(levels.numel(), generator=gen, device="cuda"))
    order[::20] = order[::20].roll(1)
    order = torch.cat((torch.tensor([levels.numel()], device="cuda"), order))
    later = torch.empty_like(order)
    later[order] = torch.arange(len(counts), device="cuda").repeat_interleave(
        torch.tensor([n // group for n in counts], device="cuda"))
    return later


def _ring(gen, levels, rows, group, heads):
    """The importance ring over ``rows`` tokens: head-summed probability rows of consecutive steps, which look alike.
    Attention goes to stretches of text, a level more or less by a factor of two; the tokens behind the last block are
    the newest."""
    of_block = -0.8 * levels + 0.3 * torch.rand(levels.numel(), generator=gen, device="cuda")
    logits = torch.zeros(RING_ROWS, rows, device="cuda")
    logits[:, :levels.numel() * group] = of_block.repeat_interleave(group)
    logits += 0.5 * torch.randn(RING_ROWS, rows, generator=gen, device="cuda")
    ring = last_attn_weights(RING_ROWS)
    ring.set_max_length(rows)
    ring.weights = (torch.softmax(logits, -1) * heads).half()
    ring.kv_seq_len = rows
    return ring


def _prefill_flush(cfg, k, v, ring, times_range):
    """Quantise all but the last ``cfg.residual`` tokens of a fresh cache."""
    flushed = cfg.context - cfg.residual
    ranked = ring.calculate_token_importance()[:flushed].clone()
    ids = get_block_token_idx(cfg.group, flushed // cfg.group, ranked)
    counts = torch.tensor(tier_counts(cfg), dtype=torch.int32)
    cache = (None,) * 39 + (k, v, cfg.context)
    return KV_cache_hqe_2(cache, flushed, 0, ids, counts, counts.clone(), ranked, cfg.strategy, None, cfg.group, cfg.group,
                          times_range)


def prepare(case, seed):
    gen = _generator(seed)
    kind, B, H = case["kind"], case["batch"], case["kv_heads"]
    state = {"case": case}
    if kind == "codec":
        state["k"], state["v"] = _kv(gen, B, H, case["tokens"])
        return state
    if kind in ("decode", "layer"):
        cfg = _config(case, case["flushed"], case["residual"], case["evict"])
        state["strategy"], state["layers"] = cfg.strategy, []
        for _ in range(case["layers"]):
            k, v = _kv(gen, B, H, cfg.context)
            ring = _ring(gen, _levels(gen, tier_counts(cfg), cfg.group), cfg.context, cfg.group, cfg.nh_q * B)
            cache = _prefill_flush(cfg, k, v, ring, False)
            q = torch.randn(B, cfg.nh_q, 1, D, generator=gen, device="cuda", dtype=torch.float16)
            layer = {"cache": cache, "q": q}
            if kind == "layer":
                layer["k"], layer["v"] = _kv(gen, B, H, 1)
                layer["ring"] = last_attn_weights(RING_ROWS)
                layer["ring"].set_max_length(cfg.context + 64)
            state["layers"].append(layer)
        return state
    # flush
    cfg = _config(case, case["history"] + case["window"], case["keep"], _share_evicted(case))
    counts = tier_counts(cfg)
    if case["history"]:
        past = _config(case, case["history"], case["window"] + case["keep"], 0.0)
        k, v = _kv(gen, B, H, past.context)
        levels = _levels(gen, tier_counts(past), past.group)
        ring = _ring(gen, levels, past.context, past.group, past.nh_q * B)
        state["cache"] = _prefill_flush(past, k, v, ring, case["times_range"])
        levels = _later_levels(gen, levels, counts, cfg.group)
    else:
        k, v = _kv(gen, B, H, cfg.context)
        state["cache"] = (None,) * 39 + (k, v, cfg.context)
        levels = _levels(gen, counts, cfg.group)
    state["ring"] = _ring(gen, levels, cfg.context, cfg.group, cfg.nh_q * B)
    state["rows"] = state["ring"].weights.clone()
    state["strategy"], state["counts"] = cfg.strategy, torch.tensor(counts, dtype=torch.int32)
    return state


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "decode":
        g = case["group"]
        return [qkv_matmul_hqe_2(layer["q"], layer["cache"], None, D, state["strategy"], g, g) for layer in state["layers"]]
    if kind == "layer":
        g, out = case["group"], []
        for layer in state["layers"]:
            cache = layer["cache"]
            new_k = torch.cat((cache[39], layer["k"]), dim=2)
            new_v = torch.cat((cache[40], layer["v"]), dim=2)
            cache = cache[:39] + (new_k, new_v, cache[41] + 1)
            weights, context = qkv_matmul_hqe_2(layer["q"], cache, None, D, state["strategy"], g, g)
            layer["ring"].update(weights)
            out.append((new_k, new_v, weights, context, layer["ring"].weights))
        return out
    if kind == "flush":
        ring, g = state["ring"], case["group"]
        ring.weights.copy_(state["rows"])   # a flush that evicts compacts the ring in place
        total = case["history"] + case["window"]
        ranked = ring.calculate_token_importance()[:total].clone()
        ids = get_block_token_idx(g, total // g, ranked)
        cache = KV_cache_hqe_2(state["cache"], case["window"], case["history"], ids, state["counts"], state["counts"].clone(),
                               ranked, state["strategy"], ring, g, g, case["times_range"])
        return list(cache) + [ids, ring.weights]
    k = state["k"].transpose(2, 3)          # K is quantised along tokens: the view of the token-major cache
    g, bit = case["group"], case["bit"]
    ck, sk, zk = uniform_group_quantize_pack_last_dim(k, g, bit)
    cv, sv, zv = uniform_group_quantize_pack_last_dim(state["v"], g, bit)
    return {"k": (ck, sk, zk, uniform_group_dequantize_unpack_last_dim(ck, sk, zk, g, bit)),
            "v": (cv, sv, zv, uniform_group_dequantize_unpack_last_dim(cv, sv, zv, g, bit))}


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _tier_bytes(counts, group):
    """Bytes of one kv head's K and V in the tiers: codes, scale and zero of every group (index lists apart)."""
    total = 0.0
    for n, bits in zip(counts[:5], (16, 8, 4, 2, 1)):
        total += 2 * n * (D * bits / 8 + (4 * D / group if bits < 16 else 0))
    return total


def work(case):
    kind, B, H = case["kind"], case["batch"], case["kv_heads"]
    if kind == "codec":
        n = 2 * B * H * D * case["tokens"]  # elements of K and V
        coded = case["bit"] / 8 + 4 / case["group"]
        return {"bytes": n * (2 + coded + coded + 2), "flops": 0.0}
    if kind in ("decode", "layer"):
        cfg = _config(case, case["flushed"], case["residual"], case["evict"])
        counts, nh_q = tier_counts(cfg), cfg.nh_q
        cached = sum(counts[:5])
        length = cached + case["residual"] + (kind == "layer")
        one = B * H * (_tier_bytes(counts, case["group"]) + 4 * D * (length - cached))   # cache, residual window
        one += 2 * 8 * cached                                     # index lists of K and V
        one += B * nh_q * (4 * D + 2 * length)                    # q, output, probabilities
        if kind == "layer":
            one += B * H * 4 * D * (length - cached)              # the window with its new row is written
            one += 2 * length                                     # importance row
        return {"bytes": one * case["layers"], "flops": 4.0 * B * nh_q * length * D * case["layers"]}
    g, keep = case["group"], case["keep"]
    total = case["history"] + case["window"]
    after = tier_counts(_config(case, total, keep, _share_evicted(case)))
    moved = B * H * (_tier_bytes(after, g) + 4 * D * (case["window"] + 2 * keep))
    if case["history"]:
        moved += B * H * _tier_bytes(tier_counts(_config(case, case["history"], 0, 0.0)), g)
    moved += 16 * (case["history"] + sum(after[:5])) + 2 * RING_ROWS * total + 8 * total
    return {"bytes": moved, "flops": 0.0}


def tolerance(case):
    if case["kind"] in ("decode", "layer"):
        # fp16 probabilities (subnormal at long contexts) and fp16 outputs of fp32-accumulated products
        return {"rel": 2e-3, "max": 2e-2}
    return "exact"
