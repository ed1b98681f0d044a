"""The tracer's quotients by the noise periods (csrc/tracer.cu, over_period): fma(zh, x, RN(zl x)) with
zh = RN(1 / y), zl = RN(1 / y - zh) equals RN(x / y) for every mantissa of x, both signs."""
import numpy as np
import pytest


@pytest.mark.parametrize("period", [0.02, 0.008, 0.003])
def test_quotient_by_a_noise_period_is_correctly_rounded(period):
    y = np.float32(period)
    zh = np.float32(1.0 / np.float64(y))
    zl = np.float32(1.0 / np.float64(y) - np.float64(zh))
    x = np.arange(1 << 23, dtype=np.uint32)
    for exponent, sign in ((127, 0), (120, 1)):
        v = (x | np.uint32(exponent << 23) | np.uint32(sign << 31)).view(np.float32)
        # the products have at most 48 bits and zl x lies 24-26 bits below zh x: the sum is exact in
        # 64 bits, and rounding it once is the fused multiply-add
        q = (np.float64(zh) * v.astype(np.float64) + (zl * v).astype(np.float64)).astype(np.float32)
        assert np.array_equal(q, v / y)
