"""A flush prepares its V side on a stream of the library's own, with events and mapped counts that the calling thread keeps:
flushes on a user's stream, in several threads, in threads that come and go, and after one that ended early; against the
oracle, bit for bit."""
import threading

import numpy as np
import pytest
import torch

from oracle import hqkv_oracle as O

pytestmark = pytest.mark.gpu
G = 32


class Work:
    """Two flushes of one cache - a prefill, then 32 more tokens with a block evicted, ring and all - and what they give."""

    def __init__(self, seed, device):
        rng = np.random.default_rng(seed)
        self.steps, want, hist = [], (None,) * 42, 0
        self.results, self.rings = [], []
        for flushed, tiers in ((1056, (1, 8, 8, 10, 6)), (32, (1, 7, 9, 10, 6))):
            total = hist + flushed
            new = [rng.standard_normal((2, 2, flushed + 9, 128)).astype(np.float16) for _ in range(2)]
            imp = (rng.random(total) * np.repeat(rng.random(total // G), G) * 8).astype(np.float16)
            rows = rng.random((20, total + 9)).astype(np.float16)
            ids = O.block_rank(G, total // G, imp)         # (divides imp by the block length, as the flush expects it)
            counts = np.array(tuple(tiers) + (0,)) * G
            counts[5] = total - counts.sum()
            ring = O.ImportanceRing(20)
            ring.weights = rows.copy()
            self.steps.append((flushed, hist, counts.tolist()) +
                              tuple(torch.from_numpy(x.copy()).to(device) for x in (new[0], new[1], ids, imp, rows)))
            want = O.flush(want[:39] + (new[0], new[1], total + 9), flushed, hist, ids, counts, counts.copy(), imp, "uniform_group",
                           ring, G, G, True)
            self.results.append(want)
            self.rings.append(ring.weights[:, :total - counts[5]])
            hist = total - int(counts[5])

    def run(self, pause=0):
        """Both flushes in the current stream, without waiting for it; the inputs are made in that stream."""
        from hqekv_b200.model.public_func import last_attn_weights
        from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
        cache, out = (None,) * 42, []
        for flushed, hist, counts, k, v, ids, imp, rows in self.steps:
            if pause:
                torch.cuda._sleep(pause)
            ring = last_attn_weights(20)
            ring.weights = rows.clone()
            cache = cache[:39] + (k.clone(), v.clone(), hist + flushed + 9)
            cache = KV_cache_hqe_2(cache, flushed, hist, ids.clone(), counts, list(counts), imp.clone(), "uniform_group", ring, G, G,
                                   True)
            # memory that the call has let go is the stream's again at once
            torch.full((1 << 21,), -1, dtype=torch.int32, device=k.device)
            out.append((cache, ring.weights))
        return out

    def check(self, out):
        for (got, ring), want, rows in zip(out, self.results, self.rings):
            for i in range(41):
                assert (got[i] is None) == (want[i] is None), i
                if want[i] is not None:
                    a = got[i].cpu().numpy()
                    assert a.shape == want[i].shape and a.tobytes() == want[i].tobytes(), i
            assert ring.cpu().numpy()[:, :rows.shape[1]].tobytes() == rows.tobytes()


def fails_early(device):
    """A flush whose K tiers do not hold whole groups: refused after both plans have been launched."""
    from hqekv_b200._lib import HqkvError
    from hqekv_b200.quant.hqe_2 import KV_cache_hqe_2
    x = torch.zeros(1, 1, 64, 128, dtype=torch.float16, device=device)
    counts = [0, 48, 16, 0, 0, 0]
    with pytest.raises(HqkvError):
        KV_cache_hqe_2((None,) * 39 + (x, x.clone(), 64), 64, 0, torch.arange(64, device=device), counts, counts,
                       torch.ones(64, dtype=torch.float16, device=device), "uniform_group")


@pytest.mark.parametrize("pause", [0, 1_000_000])          # cycles that the stream is behind the host
def test_user_stream(cuda_device, pause):
    work = Work(1, cuda_device)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        outs = [work.run(pause) for _ in range(4)]
    stream.synchronize()
    for out in outs:
        work.check(out)


def test_after_an_early_end(cuda_device):
    work = Work(2, cuda_device)
    for _ in range(3):
        fails_early(cuda_device)
        out = work.run()
        fails_early(cuda_device)
        work.check(out)


def in_threads(functions):
    errors = []

    def guarded(f):
        try:
            f()
        except BaseException as e:  # noqa: B902 - handed to the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(f,)) for f in functions]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
        assert not t.is_alive()
    if errors:
        raise errors[0]


@pytest.mark.parametrize("own_stream", [True, False])
def test_threads(cuda_device, own_stream):
    works = [Work(10 + i, cuda_device) for i in range(3)]
    torch.cuda.synchronize()

    def loop(work):
        stream = torch.cuda.Stream() if own_stream else torch.cuda.default_stream()
        with torch.cuda.stream(stream):
            for i in range(6):
                if i == 3:
                    fails_early(cuda_device)
                work.check(work.run())

    in_threads([lambda w=w: loop(w) for w in works])


def test_threads_that_come_and_go(cuda_device):
    work = Work(20, cuda_device)
    torch.cuda.synchronize()
    for _ in range(5):
        outs = []
        # the threads have ended before their results are looked at, one of them behind a flush that ended early
        in_threads([lambda: outs.append(work.run()), lambda: fails_early(cuda_device)])
        work.check(outs[0])


def test_refused_under_capture(cuda_device):
    """A flush asks the device for the tier sizes, so it cannot be captured: an error, and the next flush is as good as any."""
    work = Work(30, cuda_device)
    out = work.run()
    torch.cuda.synchronize()
    work.check(out)
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            work.run()
    torch.cuda.synchronize()
    for _ in range(2):
        work.check(work.run())
