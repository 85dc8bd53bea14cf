"""The quantiser multiplies by the fp32 reciprocal of a group's scale instead of dividing: its fp16 quotient has to be the one of
the division for every significand of the difference and of the scale, and every exponent that a code depends on."""
import numpy as np


def test_product_with_the_reciprocal_rounds_as_the_quotient():
    diff = np.arange(1024, 2048, dtype=np.float32)
    diff = np.concatenate([diff * np.float32(2.0 ** e) for e in range(-3, 9)])   # quotients from below 1/8 to above 256
    for scale in range(1024, 2048):
        product = (diff * (np.float32(1.0) / np.float32(scale))).astype(np.float16)
        quotient = (diff.astype(np.float64) / scale).astype(np.float16)  # an 11-bit result of 53 bits: rounded once
        inside = diff <= 256.0 * scale
        assert np.array_equal(product[inside], quotient[inside])
