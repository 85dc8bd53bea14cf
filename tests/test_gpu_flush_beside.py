"""The builds of a flush's two sides in the caller's stream or beside each other: sizes below and above the line between the two,
in a stream that lags behind the host and in threads; every tensor of the cache against the oracle."""
import threading

import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu
G = 32


# batch, heads, tokens of the first flush: below the line, on it, above it also with 32 more tokens into the cache, on it with two
# planes
@pytest.mark.parametrize("B,H,tokens", [(4, 8, 1248), (4, 8, 1280), (4, 8, 5120), (2, 1, 20480)])
def test_sizes(cuda_device, B, H, tokens):
    from hqekv_b200.model.public_func import last_attn_weights
    from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
    rng = np.random.default_rng(tokens)
    steps, want, hist = [], (None,) * 42, 0
    wants, rows_kept = [], []
    for flushed in (tokens, 32):
        total = hist + flushed
        k, v = (rng.standard_normal((B, H, flushed + 3, 128)).astype(np.float16) for _ in range(2))
        imp = (rng.random(total) * np.repeat(rng.random(total // G), G) * 8).astype(np.float16)
        rows = rng.random((20, total + 3)).astype(np.float16)
        ids = O.block_rank(G, total // G, imp)
        counts = np.array([int(total * f) // G * G for f in (0.05, 0.2, 0.3, 0.3)] + [0, 2 * G])
        counts[4] = total - counts.sum()
        ring = O.ImportanceRing(20)
        ring.weights = rows.copy()
        steps.append((flushed, hist, counts.tolist(), *(torch.from_numpy(x.copy()).to(cuda_device) for x in (k, v, ids, imp, rows))))
        want = O.flush(want[:39] + (k, v, total + 3), flushed, hist, ids, counts, counts.copy(), imp, "uniform_group", ring, G, G, True)
        wants.append(want)
        rows_kept.append(ring.weights[:, :total - counts[5]])
        hist = total - int(counts[5])

    def run():
        cache, out = (None,) * 42, []
        with torch.cuda.stream(torch.cuda.Stream()):
            for flushed, past, counts, k, v, ids, imp, rows in steps:
                torch.cuda._sleep(300_000)
                ring = last_attn_weights(20)
                ring.weights = rows.clone()
                cache = cache[:39] + (k.clone(), v.clone(), past + flushed + 3)
                cache = KV_cache_hqe_2(cache, flushed, past, ids.clone(), counts, list(counts), imp.clone(), "uniform_group", ring, G, G, True)
                torch.full((1 << 21,), -1, dtype=torch.int32, device=cuda_device)   # memory that the call has let go
                out.append((cache, ring.weights))
        torch.cuda.synchronize()
        results.append(out)

    results = []
    torch.cuda.synchronize()
    threads = [threading.Thread(target=run) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(results) == 2
    for out in results:
        for (got, ring), w, rows in zip(out, wants, rows_kept):
            for i in range(41):
                assert (got[i] is None) == (w[i] is None), i
                if w[i] is not None:
                    assert got[i].cpu().numpy().tobytes() == w[i].tobytes(), i
            assert ring.cpu().numpy()[:, :rows.shape[1]].tobytes() == rows.tobytes()
