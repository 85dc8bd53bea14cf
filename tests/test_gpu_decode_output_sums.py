"""The sum of the shares of a plane's outputs: as good as the fp64 sum of fp32 parts, whatever the values of V."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
LENGTH = 1 << 15


def _decode(cache, q, scratch="full"):
    """hqkv_decode_attention on the 42-slot tuple; scratch: all that is asked for, or the least that is taken."""
    from hqekv_b200._lib import check, lib, ptr, stream_ptr
    from hqekv_b200.quant._cache import build_cache_desc
    desc, keep, length, _ = build_cache_desc(cache, q.shape[1], 32, 32, 0)
    need = lib.hqkv_decode_workspace_bytes(C.byref(desc))
    if scratch == "least":  # (without the low words of the outputs)
        need -= (q.numel() * 8 + 255) & ~255
    ws = torch.zeros(need, dtype=torch.uint8, device=q.device)
    w = torch.empty(q.shape[0], q.shape[1], 1, length, dtype=torch.float16, device=q.device)
    out = torch.empty_like(q)
    check(lib.hqkv_decode_attention(C.byref(desc), ptr(q), ptr(w), ptr(out), ptr(ws), ws.numel(), stream_ptr(q.device)))
    return out


def _flat_cache(dev, kv_heads, tier, codes, scale, zero):
    """LENGTH tokens with equal logits, all in one tier and the V of a token = code * scale + zero in every channel: the
    probabilities are equal, their sum is a power of two and exact, an output is the mean of V."""
    slot, bits = {8: (4, 8), 4: (12, 4)}[tier]
    cache = [None] * 42
    idx = torch.arange(LENGTH, device=dev)
    half = dict(dtype=torch.float16, device=dev)
    cache[slot] = torch.zeros(1, kv_heads, 128, LENGTH * bits // 32, dtype=torch.int32, device=dev)
    cache[slot + 2] = torch.zeros(1, kv_heads, 128, LENGTH // 32, **half)
    cache[slot + 3] = torch.zeros(1, kv_heads, 128, LENGTH // 32, **half)
    cache[slot + 1] = cache[slot + 5] = idx
    cache[slot + 4] = torch.full((1, kv_heads, LENGTH, 128 * bits // 32), -1 if codes else 0, dtype=torch.int32, device=dev)
    for at, v in ((slot + 6, scale), (slot + 7, zero)):
        cache[at] = v.to(**half).view(1, 1, LENGTH, 1).expand(1, kv_heads, LENGTH, 4).contiguous()
    cache[41] = LENGTH
    return tuple(cache), torch.zeros(1, 4 * kv_heads, 1, 128, **half)


# kv heads: some 40, 130 and 260 or more shares a plane
@pytest.mark.parametrize("kv_heads", [8, 2, 1])
@pytest.mark.parametrize("scratch", ["full", "least"])
def test_small_parts_count(cuda_device, kv_heads, scratch):
    """One part is half of the smallest half, the others are 2^-35 of an output and less: together more than half, so the
    result is the smallest half.  (Rounded one by one to 2^-31 or 2^-33 they are lost, and the tie goes to 0.)"""
    zero = torch.zeros(LENGTH, device=cuda_device)
    zero[512::512] = 2.0 ** -20
    zero[5] = 2.0 ** -10
    cache, q = _flat_cache(cuda_device, kv_heads, 4, False, torch.ones(LENGTH, device=cuda_device), zero)
    assert torch.all(_decode(cache, q, scratch) == 2.0 ** -24)


@pytest.mark.parametrize("kv_heads", [8, 2, 1])
@pytest.mark.parametrize("scratch", ["full", "least"])
def test_large_parts_cancel(cuda_device, kv_heads, scratch):
    """Values of V of +-255 * 2^15, the first half of the tier against the second: every part is exact in fp32, the sum is 0.
    (Parts beyond 2^17 used to become infinite.)"""
    scale = torch.full((LENGTH,), 2.0 ** 15, device=cuda_device)
    scale[LENGTH // 2:] *= -1
    cache, q = _flat_cache(cuda_device, kv_heads, 8, True, scale, torch.zeros(LENGTH, device=cuda_device))
    assert torch.all(_decode(cache, q, scratch) == 0)


def test_static_scratch_takes_what_it_took(cuda_device):
    """The built-in scratch still takes a cache whose sums fit it and whose low words do not."""
    from hqekv_b200 import synthetic
    from hqekv_b200._lib import check, lib, ptr, stream_ptr
    from hqekv_b200.quant._cache import build_cache_desc
    limit = lib.hqkv_decode_static_scratch_bytes()
    cfg = synthetic.CacheConfig("", 1, 32, 8, 128, 130048 + 1024, 1024, (0.2, 0.4, 0.4), 0.0, 32, True, 1)
    cache, q = synthetic.build_cache(cfg, cuda_device, seed=3)
    for window in range(1024):
        short = cache[:39] + (cache[39][:, :, :window].contiguous(), cache[40][:, :, :window].contiguous(), 130048 + window)
        desc, keep, length, _ = build_cache_desc(short, 32, 32, 32, 0)
        need = lib.hqkv_decode_workspace_bytes(C.byref(desc))
        if need > limit:
            break
    assert need - q.numel() * 8 <= limit < need
    w = torch.empty(1, 32, 1, length, dtype=torch.float16, device=cuda_device)
    out = torch.empty_like(q)
    check(lib.hqkv_decode_attention_static(C.byref(desc), ptr(q), ptr(w), ptr(out), stream_ptr(cuda_device)))
    assert (out.float() - _decode(short, q).float()).abs().max() <= 2.0 ** -10 * out.float().abs().max()
