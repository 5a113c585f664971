"""The slot kernel divides squared costs by -0.18 (the view priors) with the
rounded reciprocal and one fused correction (Markstein).  Scaling by powers of
two commutes with every step, so one binade of numerators shows that the quotient
equals IEEE division."""
import numpy as np


def test_every_mantissa_divides_exactly():
    v = np.float32(-0.18)
    y = np.float32(1.0) / v
    a = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(0x3F800000)).view(np.float32)
    want = a / v
    q = a * y
    # exact: the products have 48 bits, and the remainder of a quotient within an ulp fits 24
    rem = a.astype(np.float64) - q.astype(np.float64) * np.float64(v)
    r = rem.astype(np.float32)
    assert np.array_equal(r.astype(np.float64), rem)
    # r y + q rounds to `want` when it is nearer than half the smaller neighbouring gap.
    # r y and q - want are exact; their sum rounds monotonically, so it can be below the
    # representable half gap only if the exact sum is.
    off = np.abs(r.astype(np.float64) * np.float64(y) + (q.astype(np.float64) - want.astype(np.float64)))
    gap = np.abs(want.astype(np.float64) - np.nextafter(want, np.float32(0)).astype(np.float64))
    assert (off < 0.5 * gap).all()
