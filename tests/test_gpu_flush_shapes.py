"""Flushes at the edges of the build kernels' tiles and runs - last tiles of one group, groups of 32, 64 and 128, one token
left in the residual window and none, evictions, groups of equal or cancelling values in the codebook tier - and rankings
on both sides of the counting kernel's limit; bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu
NORMAL = "high_uniform_group_low_normal_group"


def same(a, b, what):
    if a is None or b is None:
        assert a is None and b is None, what
        return
    a = a.cpu().numpy()
    assert a.shape == b.shape and a.dtype == b.dtype and a.tobytes() == b.tobytes(), what


# batch, kv heads, group, strategy, range in the V ranking, then per flush: tokens appended, tokens flushed, groups in the
# 16/8/4/2/1-bit tiers afterwards
@pytest.mark.parametrize("case", [
    (1, 1, 32, "uniform_group", True, ((96, 96, (0, 1, 1, 1, 0)), (32, 32, (0, 2, 1, 1, 0)))),
    (2, 2, 32, "uniform_group", False, ((545, 544, (0, 5, 5, 7, 0)), (64, 64, (0, 5, 6, 7, 0)), (31, 32, (0, 5, 6, 7, 0)))),
    (1, 2, 32, NORMAL, True, ((1075, 1056, (2, 0, 9, 9, 13)), (32, 32, (2, 0, 10, 9, 13)), (40, 32, (1, 0, 10, 8, 13)))),
    (2, 1, 64, "uniform_group", True, ((653, 640, (1, 2, 3, 4, 0)), (64, 64, (0, 3, 3, 4, 0)))),
    (1, 2, 64, NORMAL, True, ((640, 640, (1, 2, 2, 2, 3)), (65, 64, (1, 1, 2, 2, 4)))),
    (1, 1, 128, "uniform_group", False, ((1290, 1280, (0, 3, 3, 3, 1)), (128, 128, (0, 2, 3, 3, 2))))])
def test_flush_shapes(cuda_device, case):
    from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
    B, H, g, strategy, times_range, steps = case
    rng = np.random.default_rng(B + 10 * H + g)
    want, hist, got = (None,) * 42, 0, (None,) * 42
    for n, flushed, tiers in steps:
        new = []
        for slot in (39, 40):
            x = rng.standard_normal((B, H, n, 128)).astype(np.float16)
            x[:, :, :, 3] = np.float16(0.25)                                    # a constant channel
            x[:, :, :, 64:] = np.where(rng.random((B, H, n, 1)) < 0.2, np.float16(0.0), x[:, :, :, 64:])
            x[:, :, 1::2, 40] = -x[:, :, 0::2, 40][:, :, :n // 2]               # pairs that cancel
            x[:, :, :, 33:64:2] = -x[:, :, :, 32:64:2] if n % 2 else x[:, :, :, 33:64:2]
            new.append(x if want[slot] is None else np.concatenate((want[slot], x), axis=2))
        total = hist + flushed
        seq = total + new[0].shape[2] - flushed
        want, got = want[:39] + (new[0], new[1], seq), got[:39] + tuple(torch.from_numpy(x).to(cuda_device) for x in new) + (seq,)
        imp = (rng.random(total) * np.repeat(rng.random(total // g), g) * 8).astype(np.float16)
        imp_t = torch.from_numpy(imp.copy()).to(cuda_device)
        ids = O.block_rank(g, total // g, imp)
        imp_t /= g
        counts = np.array(tuple(tiers) + (0,)) * g
        counts[5] = total - counts.sum()                                        # evicted
        got = KV_cache_hqe_2(got, flushed, hist, torch.from_numpy(ids).to(cuda_device), torch.from_numpy(counts),
                             torch.from_numpy(counts.copy()), imp_t, strategy, None, g, g, times_range)
        want = O.flush(want, flushed, hist, ids, counts, counts.copy(), imp, strategy, None, g, g, times_range)
        for i in range(41):
            same(got[i], want[i], f"{flushed} tokens into {hist}: slot {i}")
        hist = total - int(counts[5])


@pytest.mark.parametrize("blocks", [1, 33, 4096, 4097])
def test_ranking_sizes(cuda_device, blocks):
    from hqekv_b200.model.public_func import get_block_token_idx
    rng = np.random.default_rng(blocks)
    imp = np.repeat(rng.integers(0, 97, blocks) / 64, 32).astype(np.float16)    # many equal keys
    imp_t = torch.from_numpy(imp.copy()).to(cuda_device)
    same(get_block_token_idx(32, blocks, imp_t), O.block_rank(32, blocks, imp), "ids")
    same(imp_t, imp, "divided importance")
