"""The two words of an output (v_finish of csrc/decode.cu) restated: whatever the order in which the shares' additions arrive, one
thread finishes the output, and what it writes is the sum of the shares."""
import math
import random
from fractions import Fraction

import numpy as np
import pytest

COUNT_AT, LOW_BITS, MARK, WORD = 52, 42, 1 << 63, (1 << 64) - 1


def count(word):
    return ((word + (1 << (COUNT_AT - 1)) & WORD) & ~(3 << 62)) >> COUNT_AT


def part(word):
    word &= (1 << COUNT_AT) - 1
    return word - (1 << COUNT_AT) if word >> (COUNT_AT - 1) else word


class Share:
    """A thread's steps, one access to memory each."""

    def __init__(self, v, bits, n):
        v, units = np.float32(v), np.float32(2.0 ** (25 - bits))
        assert abs(v) < 2.0 ** (25 + bits)
        whole = np.rint(v * units)
        rest = np.float32(np.float64(v) * np.float64(units) - np.float64(whole))   # exact: a fused multiply-add
        self.add = [(1 << COUNT_AT) + int(whole), (1 << COUNT_AT) + int(np.rint(rest * np.float32(2 ** LOW_BITS)))]
        self.n, self.steps, self.done = n, self._steps(), False

    def _steps(self):
        words = self.words
        words[1] = low = (words[1] + self.add[1]) & WORD
        yield
        words[0] = high = (words[0] + self.add[0]) & WORD
        high_done, low_done = count(high) == self.n, count(low) == self.n
        if high_done and not low_done:
            yield
            low = words[1]
            low_done = count(low) == self.n
            if not low_done:
                yield
                low = words[1]
                words[1] |= MARK
                low_done = count(low) == self.n
        elif low_done and not high_done:
            low_done = bool(low & MARK)
            if low_done:
                yield
                high = words[0]
                assert count(high) == self.n
        if low_done:
            self.out.append((high, low))


def run(values, bits, rng, swapped):
    words, out = [0, 0], []
    shares = [Share(v, bits, len(values)) for v in values]
    for s in shares:
        s.words, s.out = words, out
    live = list(shares)
    if swapped:   # the memory system takes the additions to the two words in different orders: those to the high word first
        for s in shares:
            s.add[0], s.add[1] = s.add[1], s.add[0]
    while live:
        s = rng.choice(live)
        if next(s.steps, live) is live:
            live.remove(s)
    assert len(out) == 1
    high, low = out[0]
    if swapped:
        return part(low), part(high)
    return part(high), part(low)


@pytest.mark.parametrize("n", [1, 2, 3, 7, 64, 512])
@pytest.mark.parametrize("bits", [0, 5, 15, 22])
@pytest.mark.parametrize("swapped", [False, True])
def test_one_thread_has_the_sum(n, bits, swapped):
    rng = random.Random(1000 * n + bits)
    for trial in range(200 if n < 64 else 6):
        kind = trial % 3
        values = [rng.gauss(0, 1) * (2.0 ** rng.uniform(-30, 10) if kind == 0 else 1.0) for _ in range(n)]
        if kind == 2:   # as large as they get, all of one sign or of both
            top = 2.0 ** (25 + bits) / n
            values = [top * (1 if trial % 2 else rng.choice((-1, 1))) * rng.uniform(0.9, 0.999) for _ in range(n)]
        values = [float(np.float32(v)) for v in values]
        high, low = run(values, bits, rng, swapped)
        got = (Fraction(high) + Fraction(low, 2 ** LOW_BITS)) * Fraction(2) ** (bits - 25)
        assert abs(got - sum(map(Fraction, values))) <= n * Fraction(2) ** (bits - 68)


def test_flags_stay():
    """Whatever signs are added before and after a mark of the highest bits, they and the count are what they were."""
    rng = random.Random(1)
    for n in (2, 64, 512):
        word, flag, at = 0, 0, rng.randrange(n)
        for i in range(n):
            if i == at:
                flag = rng.choice((1, 2, 3)) << 62
                word |= flag
            word = (word + (1 << COUNT_AT) - rng.randrange(1 << 40)) & WORD
        assert count(word) == n and word & (3 << 62) == flag
    assert math.log2(512 * 2 ** 41) < COUNT_AT - 1   # low words, and high ones: 2^50
