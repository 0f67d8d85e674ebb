"""Half-up rounding with a packed product in front of the +0.5.

The quantizers compute floor(RN(RN(x * s) + 0.5)).  A packed fp32 product whose only use is a packed addition may be
compiled to one fused operation, floor(RN(x * s + 0.5)).  The two differ where x * s lies just below -0.5 and the product's
rounding moves it onto -0.5.  Enumerated here: every bf16 group maximum, and for each of them every bf16 value of the
group whose product is not too small to matter, in each of the half-up modes.  No byte differs.  (Nearest-even ties do
differ, so that mode multiplies one value at a time.)
"""
import numpy as np
import pytest

F = np.float32
_BITS = np.arange(1, 0x7F80, dtype=np.uint32)          # positive finite bf16, subnormal ones included


def _factor(mode, amax):
    if mode == "fused":
        return F(127) / (amax + F(1e-5))
    amax = np.maximum(amax, F(1e-4))
    return F(127) / amax if mode == "triton" else (F(1) / amax) * F(127)


@pytest.mark.parametrize("mode", ["triton", "rowrcp", "fused"])
def test_fused_product_changes_no_half_up_byte(mode):
    with np.errstate(under="ignore"):
        s_all = _factor(mode, (_BITS << 16).view(F))
        for i in range(0, len(_BITS), 2048):
            # 10 octaves of 128 values below the maximum: |x * s| < 1/4 further down, and both forms give 0
            bits = _BITS[i:i + 2048, None].astype(np.int64) - np.arange(1280)
            x, s = (np.maximum(bits, 0).astype(np.uint32) << 16).view(F), s_all[i:i + 2048, None]
            for sign in (F(1), F(-1)):
                separate = np.floor(sign * (x * s) + F(0.5))
                fused = np.floor((sign * x.astype(np.float64) * s + 0.5).astype(F))    # 8 + 24 bits: exact before the one rounding
                assert np.array_equal(separate, fused)


def test_the_difference_exists():
    """A factor that no bf16 maximum gives: the product rounds onto -0.5 and the two forms part."""
    x, s = F(1 + 2.0 ** -7), F(0.5) / F(1 + 2.0 ** -7)
    while float(x) * float(s) <= 0.5:
        s = np.nextafter(s, F(1))
    assert float(F(x * s)) == 0.5 and np.floor(F(-(x * s)) + F(0.5)) == 0
    assert np.floor(F(-float(x) * float(s) + 0.5)) == -1
