"""The variants of the V pass (pairs of 16-token steps and warps per CTA, channel groups, heads that are there) and of the K pass
(groups of 64 and 128) at the edges of their tiles, and outputs that are not numbers; against the fp32 oracle."""
import re

import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu
CODEBOOK = "high_uniform_group_low_normal_group"
tilings = []


def _build(dev, B, nh_q, nh_kv, ctx, res, shares, f16, group, strategy, shuffled, seed=3):
    from hqekv_b200 import synthetic
    cfg = synthetic.CacheConfig("", B, nh_q, nh_kv, 128, ctx, res, shares, 0.0, group, True, 1, f16, strategy)
    cache, q = synthetic.build_cache(cfg, dev, seed=seed)
    if shuffled:
        perm = torch.randperm(ctx - res, device=dev, generator=torch.Generator(dev).manual_seed(5))
        cache = tuple(perm[x] if torch.is_tensor(x) and x.dtype == torch.int64 else x for x in cache)
    return cache, q


def _oracle(cache, q, group, strategy):
    host = tuple(x.cpu().numpy() if torch.is_tensor(x) else x for x in cache)
    return O.decode_attention(q.cpu().numpy(), host, None, group, group, quant_strategy=strategy)


# The shapes were taken so that every tiling runs (how a shape is divided is the library's affair: test_every_tiling_ran).
# (batch, query heads, kv heads, context, residual, shares, fp16 tokens, group, strategy, shuffled), GV, mode
@pytest.mark.parametrize("case,kernel", [
    ((1, 32, 8, 3 * 256 + 32 + 33, 33, (0.3, 0.4, 0.3), 0, 32, "uniform_group", False), (5, 0)),     # last tile of 32, L odd
    ((1, 16, 8, 1024 + 2, 2, (0.25, 0.25, 0.25, 0.25), 64, 32, CODEBOOK, True), (5, 1)),             # two heads, any positions
    ((1, 8, 8, 2 * 256 + 7, 7, (0.5, 0.25, 0.25), 0, 64, "uniform_group", False), (6, 1)),           # one head
    ((1, 32, 8, 32640 + 45, 45, (0.0, 0.34, 0.33, 0.33), 64, 32, CODEBOOK, False), (5, 0)),
    ((1, 32, 8, 32640 + 2, 2, (0.2, 0.4, 0.4), 0, 128, "uniform_group", True), (7, 0)),
    ((40, 32, 8, 1376 + 32 + 13, 13, (0.3, 0.4, 0.3), 0, 64, "uniform_group", False), (6, 0)),
    ((40, 16, 8, 1152 + 4, 4, (0.25, 0.25, 0.25, 0.25), 128, 128, "uniform_group", False), (7, 1)),       # 2 and 1 bits, groups of 128
    ((40, 32, 8, 1088 + 6, 6, (0.2, 0.2, 0.3, 0.3), 32, 64, CODEBOOK, True), (6, 0))])
def test_variants(cuda_device, case, kernel):
    from torch.profiler import ProfilerActivity, profile

    from hqekv_b200.quant.hqe_matmul import qkv_matmul_hqe_2
    group, strategy = case[7], case[8]
    cache, q = _build(cuda_device, *case)
    qkv_matmul_hqe_2(q, cache, None, 128, strategy, group, group)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        w, out = qkv_matmul_hqe_2(q, cache, None, 128, strategy, group, group)
        torch.cuda.synchronize()
    ran = [tuple(map(int, m.groups())) for e in prof.key_averages()
           for m in [re.search(r"v_pass_kernel<(\d+), (?:\(.*?\))?(\d+), (\d+), (\d+)>", e.key)] if m]
    assert len(ran) == 1 and ran[0][:2] == kernel, [e.key for e in prof.key_averages()]
    tilings.append(ran[0][2:])
    ow, oo = _oracle(cache, q, group, strategy)
    out, w = out.float().cpu().numpy(), w.float().cpu().numpy()
    assert float((np.abs(out - oo).max(-1) / np.abs(oo).max(-1)).max()) <= 2e-3
    assert np.all(np.abs(w - ow) <= 2.0 ** -24 + 2.0 ** -9 * ow)


def test_every_tiling_ran():
    """(pairs of steps, warps) of the calls above: if this fails, the division of work has changed and other shapes are due there."""
    if len(tilings) < 8:
        pytest.skip("follows the whole of test_variants")
    assert set(tilings) == {(1, 8), (2, 8), (2, 4)}


# shares of a plane: up to 64, more, more than 256
@pytest.mark.parametrize("case", [
    (1, 32, 8, 3072 + 40, 40, (0.3, 0.4, 0.3), 0, 32, "uniform_group", False),
    (1, 4, 1, 24 * 1024 + 40, 40, (0.3, 0.4, 0.3), 0, 32, "uniform_group", False),
    (1, 4, 1, 70 * 1024 + 40, 40, (0.3, 0.4, 0.3), 0, 32, "uniform_group", False)])
def test_outputs_that_are_not_numbers(cuda_device, case):
    from hqekv_b200.quant.hqe_matmul import qkv_matmul_hqe_2
    group, strategy = case[7], case[8]
    cache, q = _build(cuda_device, *case)
    cache = list(x.clone() if torch.is_tensor(x) else x for x in cache)
    residual = cache[40]
    residual[0, 0, 3, 5] = float("nan")
    residual[0, 0, 4, 6] = float("inf")
    residual[0, 0, 5, 7] = -float("inf")
    residual[0, 0, 6, 8], residual[0, 0, 7, 8] = float("inf"), -float("inf")
    residual[0, 0, :, 9] = 65504.0                      # the largest number, with both signs, in what is not quantised
    residual[0, 0, ::2, 9] = -65504.0
    if case[2] > 1:  # 8-bit values beyond the range of fp16 in some channels of the second and third head
        cache[10][0, 1, :, 0] = 6e4
        cache[10][0, 2, :, 1] = -6e4
    cache = tuple(cache)
    _, out = qkv_matmul_hqe_2(q, cache, None, 128, strategy, group, group)
    with np.errstate(all="ignore"):
        want = _oracle(cache, q, group, strategy)[1].astype(np.float16).astype(np.float32)
    out = out.float().cpu().numpy()
    assert np.isnan(out[0, 0, 0, 5]) and out[0, 0, 0, 6] == np.inf and out[0, 0, 0, 7] == -np.inf and np.isnan(out[0, 0, 0, 8])
    assert np.array_equal(np.isnan(out), np.isnan(want))
    odd = ~np.isfinite(want)
    assert np.array_equal(out[odd & ~np.isnan(want)], want[odd & ~np.isnan(want)])
    if case[2] > 1:
        assert np.all(out[0, 4:8, 0, :32] == np.inf) and np.all(out[0, 8:12, 0, 32:64] == -np.inf)
    error = np.where(odd, 0.0, np.abs(np.where(odd, 0.0, out) - np.where(odd, 0.0, want)))
    assert float((error.max(-1) / np.where(odd, 0.0, np.abs(np.where(odd, 0, want))).max(-1)).max()) <= 2e-3
