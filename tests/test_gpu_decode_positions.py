"""Where the tokens of a cache stand does not change what a decode computes: the same tiers with other index lists give the same
outputs and the same probabilities at other places, bit for bit.  Quads of consecutive positions (from a multiple of four on) are
read and written as such, everything else token by token; weights given by the caller likewise."""
import pytest
import torch

pytestmark = pytest.mark.gpu
STRATEGY = "high_uniform_group_low_normal_group"   # (the one that the product with given weights reads its 1-bit tier in)


def _cache(dev, nh_q, nh_kv, batch, ctx, res, group):
    from hqekv_b200 import synthetic
    cfg = synthetic.CacheConfig("", batch, nh_q, nh_kv, 128, ctx, res, (0.25, 0.25, 0.25, 0.25), 0.0, group, True, 1, 64, STRATEGY)
    return synthetic.build_cache(cfg, dev, seed=11)


def _order(kind, n, dev):
    """The new position of every old one."""
    if kind == "consecutive":      # not on multiples of four
        return torch.arange(n, device=dev).roll(2)
    if kind == "any":
        return torch.randperm(n, device=dev, generator=torch.Generator(dev).manual_seed(5))
    order = torch.arange(n, device=dev)   # all but a few are quads
    order[[3, 38, 71]] = order[[71, 3, 38]]
    return order


# (query heads, kv heads, batch): one, two, four and eight query heads per kv head; tiles of 32 and of 64 tokens, CTAs of eight and of four warps
@pytest.mark.parametrize("heads", [(8, 8, 1), (16, 8, 1), (32, 8, 1), (16, 2, 1), (8, 8, 40), (16, 8, 40), (32, 8, 40)])
@pytest.mark.parametrize("ctx,res", [(1408 + 64 + 3, 3), (1376 + 4, 4)])   # rows of odd length; on 8-byte boundaries
@pytest.mark.parametrize("kind", ["consecutive", "any", "few"])
def test_positions(cuda_device, heads, ctx, res, kind):
    from hqekv_b200.quant import matmul as mm
    from hqekv_b200.quant.hqe_matmul import qkv_matmul_hqe_2
    nh_q, nh_kv, batch = heads
    cache, q = _cache(cuda_device, nh_q, nh_kv, batch, ctx, res, 32)
    order = _order(kind, ctx - res, cuda_device)
    moved = tuple(order[x] if torch.is_tensor(x) and x.dtype == torch.int64 else x for x in cache)
    place = torch.cat((order, torch.arange(ctx - res, ctx, device=cuda_device)))
    w, out = qkv_matmul_hqe_2(q, cache, None, 128, STRATEGY, 32, 32)
    w2, out2 = qkv_matmul_hqe_2(q, moved, None, 128, STRATEGY, 32, 32)
    assert torch.equal(out, out2) and torch.equal(w, w2[..., place])

    def given(tiers, weights):
        args = [tiers[2], tiers[3]]
        for s in (8, 16, 24, 32):
            args += [tiers[s], tiers[s + 1], tiers[s + 2], tiers[s + 3]]
        return mm.cuda_bmm_forward_wv_group_hq(32, nh_kv, weights, *args, tiers[40])
    mine = torch.randn(w.shape, device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(6)).half()
    there = torch.empty_like(mine)
    there[..., place] = mine
    assert torch.equal(given(cache, mine), given(moved, there))
    # the decode's own weights: the same product but for 2^-11 of every weight, which meets values of V up to some eight times the outputs
    assert (given(cache, w).float() - out.float()).abs().max() <= 4e-3 * out.float().abs().max()
