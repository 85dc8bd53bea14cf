"""Logits do not depend on how the scales of K are laid out: groups of 64 and 128, or of 32 with every scale that often."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [64, 128])
@pytest.mark.parametrize("shares", [(1.0, 0.0, 0.0, 0.0), (0.0, 1.0, 0.0, 0.0), (0.0, 0.0, 1.0, 0.0), (0.0, 0.0, 0.0, 1.0)])
def test_repeated_scales(cuda_device, group, shares):
    from hqekv_b200 import synthetic
    from hqekv_b200.quant.hqe_matmul import qkv_matmul_hqe_2
    cfg = synthetic.CacheConfig("", 4, 32, 8, 128, 4096 + 21, 21, shares, 0.0, group, True, 1, 0, "uniform_group")
    cache, q = synthetic.build_cache(cfg, cuda_device, seed=7)
    fine = list(cache)
    for k in (4, 12, 20, 28):  # K of the 8-, 4-, 2- and 1-bit tier: codes, positions, scales, zeros
        if cache[k] is not None:
            for at in (k + 2, k + 3):
                fine[at] = cache[at].repeat_interleave(group // 32, dim=-1)
    weights, out = qkv_matmul_hqe_2(q, cache, None, 128, "uniform_group", group, group)
    again, also = qkv_matmul_hqe_2(q, tuple(fine), None, 128, "uniform_group", 32, group)
    assert torch.equal(weights, again) and torch.equal(out, also)
