"""The column quantiser's ways of loading and storing a tile: rows of 128 elements and others, whole and ragged tiles, outputs on
and off the boundaries of its wide stores, and values of every magnitude; bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bit,group", [(8, 32), (4, 32), (4, 64), (2, 64), (1, 128), (1, 32)])
@pytest.mark.parametrize("tokens,channels,pitch,skip", [
    (256, 128, 128, 0),    # whole tiles, everything in wide stores
    (256, 128, 128, 1),    # outputs one element off
    (384, 72, 128, 0),     # part of a row
    (128, 200, 208, 0),    # two tiles of channels, another distance between the tokens
    (512, 2, 2, 4),        # outputs on the next boundary
    (512, 128, 136, 0)])
def test_columns(cuda_device, bit, group, tokens, channels, pitch, skip):
    _check(cuda_device, bit, group, tokens, channels, pitch, skip)


@pytest.mark.parametrize("bit,group,tokens", [(4, 32, 32), (8, 32, 160), (2, 64, 192), (4, 64, 320), (1, 32, 96), (8, 64, 64)])
def test_ragged_tokens(cuda_device, bit, group, tokens):
    _check(cuda_device, bit, group, tokens, 128, 128, 0)


def _check(dev, bit, group, tokens, channels, pitch, skip):
    from hqekv_b200._lib import check, lib, ptr, stream_ptr
    rng = np.random.default_rng(tokens + bit)
    outer = 2
    buf = rng.standard_normal((outer, tokens, pitch)).astype(np.float32)
    buf *= 2.0 ** rng.integers(-14, 13, (1, 1, pitch))   # scales from subnormal ones up
    buf = buf.astype(np.float16)
    buf[:, :, 1] = -0.75                                 # constant groups
    x = torch.from_numpy(buf).to(dev)
    rows = outer * channels
    code = torch.zeros(rows * tokens * bit // 32 + skip, dtype=torch.int32, device=dev)[skip:]
    scale, low = (torch.zeros(rows * tokens // group + skip, dtype=torch.float16, device=dev)[skip:] for _ in range(2))
    check(lib.hqkv_quantize_pack(ptr(x), rows, tokens, channels, tokens * pitch, 1, pitch, group, bit, ptr(code), ptr(scale), ptr(low),
                                 stream_ptr(x.device)))
    want = O.quantize_pack_last_dim(np.ascontiguousarray(np.swapaxes(buf[None, :, :, :channels], 2, 3)), group, bit)
    for got, w in zip((code, scale, low), want):
        assert got.cpu().numpy().tobytes() == w.tobytes()
