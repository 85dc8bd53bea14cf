"""Where the tensors of a flush may lie: tiers, residual windows and (C ABI) outputs that start on no more than their type's
own boundary, bit for bit against the oracle and against the flush of aligned tensors; and ranked ids that split blocks."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu
UNIFORM, NORMAL = "uniform_group", "high_uniform_group_low_normal_group"


def off(t):
    """The same contiguous tensor one element behind a 512-byte boundary."""
    if not torch.is_tensor(t) or t.dtype == torch.int64:
        return t
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


def same(a, b, what):
    if a is None or b is None:
        assert a is None and b is None, what
        return
    a = a.cpu().numpy()
    assert a.shape == b.shape and a.dtype == b.dtype and a.tobytes() == b.tobytes(), what


def window(rng, B, H, n):
    x = rng.standard_normal((B, H, n, 128)).astype(np.float16)
    x[:, :, :, 3] = np.float16(0.25)                       # a constant channel
    x[:, :, ::3, 64:] = np.float16(0.0)
    return x


# batch, kv heads, group, strategy, then per flush: tokens flushed (five more stay), groups in the tiers afterwards
CASES = [
    (1, 2, 32, UNIFORM, ((544, (2, 4, 5, 6, 0)), (32, (1, 5, 5, 7, 0)), (64, (1, 4, 6, 8, 0)))),
    (2, 1, 32, NORMAL, ((992, (2, 0, 9, 9, 11)), (32, (2, 0, 8, 10, 12)))),
    (1, 2, 64, NORMAL, ((640, (1, 2, 2, 2, 3)), (64, (1, 1, 2, 2, 4)))),
    (1, 1, 128, UNIFORM, ((1280, (1, 2, 3, 3, 1)), (128, (1, 2, 2, 3, 2))))]


@pytest.mark.parametrize("case", CASES)
def test_tiers_and_window_on_their_types_boundaries(cuda_device, case):
    from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
    B, H, g, strategy, steps = case
    rng = np.random.default_rng(B + 10 * H + g)
    want, got, hist = (None,) * 42, (None,) * 42, 0
    for flushed, tiers in steps:
        total = hist + flushed
        new = [window(rng, B, H, flushed + 5) for _ in range(2)]
        want = want[:39] + (new[0], new[1], total + 5)
        got = got[:39] + tuple(torch.from_numpy(x).to(cuda_device) for x in new) + (total + 5,)
        got = tuple(off(t) for t in got)
        imp = (rng.random(total) * np.repeat(rng.random(total // g), g) * 8).astype(np.float16)
        imp_t = off(torch.from_numpy(imp.copy()).to(cuda_device))
        ids = O.block_rank(g, total // g, imp)
        imp_t /= g
        counts = np.array(tuple(tiers) + (0,)) * g
        counts[5] = total - counts.sum()                   # evicted
        got = KV_cache_hqe_2(got, flushed, hist, torch.from_numpy(ids).to(cuda_device), torch.from_numpy(counts),
                             torch.from_numpy(counts.copy()), imp_t, strategy, None, g, g, True)
        want = O.flush(want, flushed, hist, ids, counts, counts.copy(), imp, strategy, None, g, g, True)
        for i in range(41):
            same(got[i], want[i], f"{flushed} tokens into {hist}: slot {i}")
        hist = total - int(counts[5])


@pytest.mark.parametrize("case", CASES)
def test_outputs_on_their_types_boundaries(cuda_device, case):
    """Plan and build of one tier at a time through the C ABI, with outputs and plan scratch on their types' boundaries."""
    from hqekv_b200._lib import CODEC_NORMAL, CODEC_UNIFORM, check, lib, ptr, stream_ptr
    from hqekv_b200.model.public_func import get_block_token_idx
    from hqekv_b200.quant._cache import build_flush_src, void_p_array
    from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
    B, H, g, strategy, steps = case
    rng = np.random.default_rng(B + 20 * H + g)
    cache, hist, st = (None,) * 42, 0, stream_ptr(cuda_device)
    for flushed, tiers in steps:
        total = hist + flushed
        new = [torch.from_numpy(window(rng, B, H, flushed)).to(cuda_device) for _ in range(2)]
        cache = cache[:39] + (new[0], new[1], total)
        imp = torch.from_numpy(rng.random(total).astype(np.float16)).to(cuda_device)
        k_ids = torch.from_numpy(O.block_rank(g, total // g, imp.cpu().numpy())).to(cuda_device)
        v_ids = get_block_token_idx(g, total // g, imp.clone())   # as the flush ranks V without value ranges
        counts = [t * g for t in tiers]
        counts.append(total - sum(counts))
        after = KV_cache_hqe_2(cache, flushed, hist, k_ids, counts, list(counts), imp, strategy, None, g, g, False)
        for side, slots, ids, build in (("K", (0, 4, 12, 20, 28), k_ids, lib.hqkv_flush_build_k),
                                        ("V", (2, 8, 16, 24, 32), v_ids, lib.hqkv_flush_build_v)):
            idx = [cache[s + 1] for s in slots]
            plan_src = torch.empty(5, total, dtype=torch.int32, device=cuda_device)
            plan_ids = torch.empty(5, total, dtype=torch.int64, device=cuda_device)
            surv = torch.empty(total, dtype=torch.int64, device=cuda_device)
            n = torch.zeros(8, dtype=torch.int32, device=cuda_device)
            ws = torch.empty(lib.hqkv_flush_plan_workspace_bytes(total) + 4, dtype=torch.uint8, device=cuda_device)[4:]
            check(lib.hqkv_flush_plan(void_p_array(idx), (C.c_int32 * 5)(*[0 if i is None else i.numel() for i in idx]), hist,
                                      flushed, ptr(ids), (C.c_int64 * 6)(*np.cumsum(counts)), ptr(plan_src), ptr(plan_ids),
                                      ptr(surv), ptr(n), ptr(ws), ws.numel(), st))
            n = n.tolist()
            src, keep = build_flush_src(cache, side, new[side == "V"], CODEC_NORMAL if strategy == NORMAL else CODEC_UNIFORM)
            for t, s in enumerate(slots):
                assert n[t] == (0 if after[s] is None else after[s + 1].numel())
                if n[t] == 0:
                    continue
                want = (after[s], after[s + 2], after[s + 3]) if t else (after[s], None, None)
                outs = [None if x is None else off(torch.zeros_like(x)) for x in want]
                check(build(src, B, H, 128, g, t, ptr(plan_src[t]), n[t], *map(ptr, outs), st))
                for x, y in zip(outs, want):
                    assert x is None or torch.equal(x.view(torch.uint8), y.view(torch.uint8)), (side, t)
                assert torch.equal(plan_ids[t, :n[t]], after[s + 1])
            del keep
        cache, hist = after[:39] + (None, None, total), total - counts[5]


@pytest.mark.parametrize("g,strategy,low,idx", [(32, UNIFORM, 3, 21), (64, NORMAL, 4, 29)])
def test_ranked_ids_that_split_blocks(cuda_device, g, strategy, low, idx):
    """Not a call that makes sense - K is quantised in blocks - but its positions are the caller's and must not send a wide
    access off its boundary or out of a tier.  The id lists are those of the plan all the same."""
    from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
    rng = np.random.default_rng(5)
    new = [torch.from_numpy(window(rng, 1, 1, 5 * g)).to(cuda_device) for _ in range(2)]
    imp = torch.ones(5 * g, dtype=torch.float16, device=cuda_device)
    counts = [0, 2 * g, 2 * g, 0, 0, 0]
    cache = (None,) * 39 + tuple(x[:, :, :4 * g].contiguous() for x in new) + (4 * g,)
    cache = KV_cache_hqe_2(cache, 4 * g, 0, torch.arange(4 * g, device=cuda_device), counts, list(counts), imp[:4 * g].clone(),
                           strategy, None, g, g)
    cache = cache[:39] + tuple(x[:, :, 4 * g:].contiguous() for x in new) + (5 * g,)
    keep = np.sort(rng.permutation(2 * g)[:g])            # half of the 8-bit tier, any tokens; the rest goes to the low tier
    rest = np.setdiff1d(np.arange(5 * g), keep)
    ids = torch.from_numpy(np.concatenate((keep, rest))).to(cuda_device)
    k_counts, v_counts = [0, g, 0, 0, 0, 0], [0, 2 * g, 0, 0, 0, 0]
    k_counts[low], v_counts[low] = 4 * g, 3 * g
    got = KV_cache_hqe_2(cache, g, 4 * g, ids, k_counts, v_counts, imp, strategy, None, g, g)
    assert got[5].tolist() == keep.tolist() and sorted(got[idx].tolist()) == rest.tolist()
    assert got[4].shape == (1, 1, 128, g // 4) and float(torch.ones(8, device=cuda_device).sum()) == 8.0
