"""The V pass alone, as often as wanted after one K pass: every call writes the outputs."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


# shares of a plane: some 40; more than 512, whose sums the last CTA reads
@pytest.mark.parametrize("heads,kv_heads,context", [(32, 8, 8192 + 40), (4, 1, 192 * 1024 + 40)])
def test_v_pass_again(cuda_device, heads, kv_heads, context):
    from hqekv_b200 import synthetic
    from hqekv_b200._lib import check, lib, ptr, stream_ptr
    from hqekv_b200.quant._cache import build_cache_desc
    cfg = synthetic.CacheConfig("", 1, heads, kv_heads, 128, context, 40, (0.3, 0.4, 0.3), 0.0, 32, True, 1)
    cache, q = synthetic.build_cache(cfg, cuda_device, seed=3)
    desc, keep, length, _ = build_cache_desc(cache, heads, 32, 32, 0)
    ws = torch.zeros(lib.hqkv_decode_workspace_bytes(C.byref(desc)), dtype=torch.uint8, device=cuda_device)

    def call(phases):
        w = torch.full((1, heads, 1, length), 7.0, dtype=torch.float16, device=cuda_device)
        out = torch.full_like(q, 7.0)
        check(lib.hqkv_decode_attention_phases(C.byref(desc), ptr(q), ptr(w), ptr(out), ptr(ws), ws.numel(), phases,
                                               stream_ptr(cuda_device)))
        return w, out

    w, out = call(3)
    for _ in range(3):
        again_w, again = call(2)
        assert torch.equal(again_w, w)
        assert torch.allclose(again.float(), out.float(), rtol=2.0 ** -10, atol=2.0 ** -24)   # (fp64 sums may fall either way)
    call(1)
    assert torch.allclose(call(2)[1].float(), out.float(), rtol=2.0 ** -10, atol=2.0 ** -24)
