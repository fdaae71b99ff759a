"""The quotient steps of the regression kernel's taps (csrc/regression.cu,
reciprocal() and quotient()), emulated in extended precision: whatever
reciprocal within 1 ulp the hardware returns, one Newton step and one residual
correction give the IEEE quotient."""
import numpy as np
import pytest

f32 = np.float32


def fma(a, b, c):
    # the product of two floats is exact in 64 bits of significand
    return (a.astype(np.longdouble) * b.astype(np.longdouble) + c.astype(np.longdouble)).astype(f32)


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs 80-bit extended precision")
@pytest.mark.parametrize("lo_a,hi_a,lo_b,hi_b", [(-40, 20, -14, 14), (-20, 99, -14, 99), (-10, 7, -7, 7)])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_quotient_is_ieee(lo_a, hi_a, lo_b, hi_b, off):
    rng = np.random.default_rng(100 + off)
    n = 400_000
    a = (rng.choice([-1.0, 1.0], n) * np.exp2(rng.uniform(lo_a, hi_a, n))).astype(f32)
    b = np.exp2(rng.uniform(lo_b, hi_b, n)).astype(f32)
    b[::8] = (b[::8].view(np.int32) | 0x7FFFFF).view(f32)   # all-ones significands
    y = (np.float64(1) / b.astype(np.float64)).astype(f32)
    y = (y.view(np.int32) + off).view(f32)
    y = fma(y, fma(-b, y, np.ones_like(b)), y)
    q = (a.astype(np.float64) * y.astype(np.float64)).astype(f32)   # exact product, rounded once
    q = fma(fma(-q, b, a), y, q)
    np.testing.assert_array_equal(q, a / b)
