"""The parts of a large tier are allocations of their own, those of a small one share one; values as the codec gives them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,apart", [(4096, False), (139264, True)])   # codes of 4 and 143 MB
def test_allocations_of_a_tier(cuda_device, tokens, apart):
    from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
    from hqekv_b200.quant.pack_unpack import uniform_group_quantize_pack_last_dim
    gen = torch.Generator(cuda_device).manual_seed(1)
    k, v = (torch.randn(1, 8, tokens, 128, generator=gen, device=cuda_device, dtype=torch.float16) for _ in range(2))
    counts = [0, tokens, 0, 0, 0, 0]
    ids = torch.arange(tokens, device=cuda_device)
    imp = torch.ones(tokens, dtype=torch.float16, device=cuda_device)
    got = KV_cache_hqe_2((None,) * 39 + (k, v, tokens), tokens, 0, ids, counts, list(counts), imp, "uniform_group")
    for first, source in ((4, k.transpose(2, 3)), (8, v)):
        parts = [got[first], got[first + 2], got[first + 3]]
        assert got[first + 1].tolist() == list(range(tokens))
        for a, b in zip(parts, uniform_group_quantize_pack_last_dim(source, 32, 8)):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
        assert len({x.untyped_storage().data_ptr() for x in parts + [got[first + 1]]}) == (4 if apart else 1)
