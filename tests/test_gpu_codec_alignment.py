"""The codec on addresses that its wide loads and stores cannot use, and on the edges of its tiles; bit-exact against the
oracle."""
import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skip", [0, 1, 8])            # halfs: 32-byte, 2-byte and 16-byte boundaries
@pytest.mark.parametrize("bit", [8, 4, 2, 1])
@pytest.mark.parametrize("group,groups", [(32, 5), (64, 3), (128, 1)])
def test_alignment(cuda_device, group, groups, bit, skip):
    from hqekv_b200.quant.pack_unpack import uniform_group_dequantize_unpack_last_dim as unpack
    from hqekv_b200.quant.pack_unpack import uniform_group_quantize_pack_last_dim as pack
    rng = np.random.default_rng(group + bit)
    shape = (2, 1, groups * group, 66)                 # token-major K: two channels beyond a warp's
    x = (rng.standard_normal(shape) * 3).astype(np.float16)
    x[0, 0, :, 5] = 1.5                                # a constant group: scale 0
    flat = torch.zeros(x.size + skip, dtype=torch.float16, device=cuda_device)
    flat[skip:] = torch.from_numpy(x.ravel()).to(cuda_device)
    for xt, xn in ((flat[skip:].view(shape).transpose(2, 3), np.ascontiguousarray(np.swapaxes(x, 2, 3))),
                   (flat[skip:].view(2, 66, 1, groups * group), x.reshape(2, 66, 1, groups * group))):
        want = O.quantize_pack_last_dim(xn, group, bit)
        code, scale, mn = pack(xt, group, bit)
        for a, b in zip((code, scale, mn), want):
            assert a.cpu().numpy().tobytes() == b.tobytes()
        words = torch.zeros(code.numel() + 1, dtype=code.dtype, device=cuda_device)
        words[1:] = code.reshape(-1)
        for c in (code, words[1:].view(code.shape)):   # packed words on any 4-byte boundary
            assert unpack(c, scale, mn, group, bit).cpu().numpy().tobytes() == O.dequantize_unpack_last_dim(*want, group, bit).tobytes()
