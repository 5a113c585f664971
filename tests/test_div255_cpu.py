"""The slot kernel divides the blur samples by 255 with the rounded reciprocal
and one fused correction (division by a constant, Brisebarre and Muller).  The
samples are k / 256 with 0 <= k < 2^16: every quotient equals IEEE division."""
from fractions import Fraction

import numpy as np


def _round32(x: Fraction, near: np.float32) -> np.float32:
    """x rounded to single precision, ties to even; near is within an ulp of it."""
    c = sorted({float(np.nextafter(near, np.float32(-1))), float(near), float(np.nextafter(near, np.float32(1e9)))})
    return np.float32(min(c, key=lambda v: (abs(Fraction(v) - x), int(np.float32(v).view(np.uint32)) & 1)))


def test_every_blur_sample_divides_exactly():
    r = np.float32(float.fromhex("0x1.010102p-8"))
    sb = (np.arange(1 << 16, dtype=np.float64) / 256.0).astype(np.float32)
    want = sb / np.float32(255.0)
    q = sb * r
    rem = (sb.astype(np.float64) - q.astype(np.float64) * 255.0).astype(np.float32)     # exact in 64 bits, then rounded
    for i in range(1 << 16):
        exact = Fraction(float(rem[i])) * Fraction(float(r)) + Fraction(float(q[i]))
        assert _round32(exact, want[i]) == want[i], f"k = {i}"
