"""Value ranges of rows that lie far apart, against the oracle, bit for bit."""
import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu


def test_rows_of_a_value_range_far_apart(cuda_device):
    """Batch entries 64 GiB and 16 bytes apart: the offset in units of 16 bytes does not fit 32 bits."""
    from hqekv_b200.model.public_func import calculate_token_range
    gap = 2 ** 35 + 8                                      # halfs
    if torch.cuda.mem_get_info()[0] < 2 * gap + 2 ** 31:
        pytest.skip("needs 66 GiB")
    base = torch.empty(gap + 2 ** 20, dtype=torch.float16, device=cuda_device)
    rng = np.random.default_rng(9)
    x = rng.standard_normal((2, 2, 33, 128)).astype(np.float16)
    v = base.as_strided((2, 2, 33, 128), (gap, 33 * 128, 128, 1))
    base[:2 ** 20] = 0.0
    v.copy_(torch.from_numpy(x).to(cuda_device))
    try:
        got = calculate_token_range(v, None).cpu().numpy()
        assert got.tobytes() == O.token_range(x).tobytes()
    finally:
        del v, base
        torch.cuda.empty_cache()
