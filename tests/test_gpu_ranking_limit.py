"""The ranking on both sides of the number of blocks where it changes from counting to sorting, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [3072, 3073, 8192])
def test_ranking_limit(cuda_device, blocks):
    from hqekv_b200.model.public_func import get_block_token_idx
    rng = np.random.default_rng(blocks)
    imp = np.repeat(rng.integers(0, 97, blocks) / 64, 32).astype(np.float16)    # many equal keys
    imp_t = torch.from_numpy(imp.copy()).to(cuda_device)
    ids = get_block_token_idx(32, blocks, imp_t).cpu().numpy()
    assert ids.tobytes() == O.block_rank(32, blocks, imp).tobytes()
    assert imp_t.cpu().numpy().tobytes() == imp.tobytes()
