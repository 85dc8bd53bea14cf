"""How the decode kernels share a plane's tokens out: CTAs that walk several tiers (many planes), CTAs of one tier, ragged
last units, positions in any order, one to eight query heads per kv head; against the fp32 oracle."""
import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu
NORMAL = "high_uniform_group_low_normal_group"


# batch, query heads, kv heads, context, residual, shares, fp16 tokens, group, strategy, shuffled positions
@pytest.mark.parametrize("case", [
    (40, 32, 8, 1376 + 13, 13, (0.3, 0.4, 0.3), 0, 32, "uniform_group", False),       # a CTA per plane, all tiers
    (64, 16, 8, 1056 + 1, 1, (0.25, 0.25, 0.25, 0.25), 64, 32, NORMAL, False),         # ... with fp16 and 1-bit tiers
    (24, 64, 8, 1536 + 70, 70, (0.25, 0.5, 0.25), 0, 64, "uniform_group", False),      # eight query heads: two CTAs
    (12, 32, 8, 4224 + 64, 64, (0.1, 0.3, 0.6), 0, 128, "uniform_group", False),       # shares that end inside tiers
    (40, 8, 8, 992 + 33, 33, (0.3, 0.4, 0.3), 0, 32, "uniform_group", True),           # one query head, any positions
    (1, 32, 8, 2080 + 5, 5, (0.2, 0.4, 0.4), 64, 32, "uniform_group", True),           # one tier per CTA, any positions
    (1, 16, 8, 96 + 100, 100, (0.34, 0.33, 0.33), 0, 32, "uniform_group", False)])     # units far from full
def test_shares(cuda_device, case):
    from hqekv_b200 import synthetic
    from hqekv_b200.quant.hqe_matmul import qkv_matmul_hqe_2
    B, nh_q, nh_kv, ctx, res, shares, f16, group, strategy, shuffled = case
    cfg = synthetic.CacheConfig("", B, nh_q, nh_kv, 128, ctx, res, shares, 0.0, group, True, 1, f16, strategy)
    cache, q = synthetic.build_cache(cfg, cuda_device, seed=11)
    if shuffled:  # the same tokens at other logical positions, the same ones for K and V
        perm = torch.randperm(ctx - res, device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(5))
        cache = tuple(perm[x] if torch.is_tensor(x) and x.dtype == torch.int64 else x for x in cache)
    w, out = qkv_matmul_hqe_2(q, cache, None, 128, strategy, group, group)
    host = tuple(x.cpu().numpy() if torch.is_tensor(x) else x for x in cache)
    ow, oo = O.decode_attention(q.cpu().numpy(), host, None, group, group, quant_strategy=strategy)
    out, w = out.float().cpu().numpy(), w.float().cpu().numpy()
    assert float((np.abs(out - oo).max(-1) / np.abs(oo).max(-1)).max()) <= 2e-3
    assert np.all(np.abs(w - ow) <= 2.0 ** -24 + 2.0 ** -9 * ow)
