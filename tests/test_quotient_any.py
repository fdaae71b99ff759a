"""The quotient of the regression kernel's repeated windows (csrc/regression.cu,
quotient_any()), emulated: the IEEE quotient for every kind of numerator and
every divisor that a tap can have (1e-4 or more, infinite, or not a number)."""
import numpy as np
import pytest

f32 = np.float32
MAX = f32(2.0) ** 100


def fma(a, b, c):
    # the product of two floats is exact in 64 bits of significand
    return (a.astype(np.longdouble) * b.astype(np.longdouble) + c.astype(np.longdouble)).astype(f32)


def reciprocal(b):
    y = (np.float64(1) / b.astype(np.float64)).astype(f32)
    return fma(y, fma(-b, y, np.ones_like(b)), y)


def quotient(a, b, y):
    q = (a.astype(np.float64) * y.astype(np.float64)).astype(f32)
    return fma(fma(-q, b, a), y, q)


def quotient_any(a, b):
    with np.errstate(all="ignore"):
        fast = (np.abs(a) < MAX) & (b < MAX)
        b_finite = b < np.inf
        both = (np.abs(a) < np.inf) & b_finite
        q = quotient(a, b, reciprocal(b))
        return np.where(fast, q, np.where(both, a / b, np.where(b_finite, a, a * (f32(1) / b))))


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs 80-bit extended precision")
def test_every_kind_of_operand():
    rng = np.random.default_rng(5)
    special = np.array([0, -0.0, 1, -3, 2.0 ** 99, 2.0 ** 100, -(2.0 ** 100), 1e34, 3e38, np.inf, -np.inf, np.nan], f32)
    div = np.array([1e-4, 1e-2, 1, 3, 2.0 ** 50, 2.0 ** 99, 2.0 ** 100, 1e34, 2.0 ** 127, 3e38, np.inf, np.nan], f32)
    a = np.concatenate([special, (rng.choice([-1, 1], 400) * np.exp2(rng.uniform(-40, 128, 400))).astype(f32)])
    b = np.concatenate([div, np.exp2(rng.uniform(-13, 128, 400)).astype(f32)])
    A, B = [np.ascontiguousarray(v.ravel()) for v in np.meshgrid(a, b)]
    with np.errstate(all="ignore"):
        want = A / B
    # quotients below the normal range are not exact in the fast form and not in question here
    keep = ~((np.abs(want) < np.finfo(f32).tiny) & (want != 0))
    np.testing.assert_array_equal(quotient_any(A, B)[keep], want[keep])
