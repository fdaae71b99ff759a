"""The quotient of the regression kernel's repeated windows (csrc/regression.cu,
quotient_any()), emulated: the IEEE quotient for every kind of numerator and
every divisor that a tap can have (1e-4 or more, infinite, or not a number)."""
import numpy as np
import pytest

f32 = np.float32
MAX = f32(2.0) ** 100


def fma(a, b, c):
    """Rounded once: the product is exact in a double, the sum is rounded to
    odd there (its error tells which way), and then to float."""
    p, c = a.astype(np.float64) * b.astype(np.float64), c.astype(np.float64)
    s = np.ascontiguousarray(p + c)
    t = s - p
    err = (p - (s - t)) + (c - t)
    bits = s.view(np.int64)
    fix = np.isfinite(s) & (err != 0) & (bits & 1 == 0)
    bits[fix] += np.where((err[fix] > 0) == (s[fix] > 0), 1, -1)
    return s.astype(f32)


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


def neighbour(b, above):
    """The float next to 1 / b on one side: what an approximation good to an ulp may return."""
    exact = np.longdouble(1) / b.astype(np.longdouble)
    y = (np.float64(1) / b.astype(np.float64)).astype(f32)
    low = np.where(y.astype(np.longdouble) > exact, np.nextafter(y, f32(0)), y)
    return np.where(low.astype(np.longdouble) == exact, low, np.nextafter(low, f32(np.inf))) if above else low


@pytest.mark.parametrize("above", [False, True])
def test_reciprocal_is_rounded_to_nearest(above):
    """Over every significand, from either neighbour: the condition under which
    the quotient's theorem holds.  The one exception is the all-ones significand
    from below; the hardware's approximation of that one is the neighbour above."""
    for part in np.array_split(np.arange(1 << 23, dtype=np.int32), 8):
        b = (part | 0x3F800000).view(f32)
        y = neighbour(b, above)
        y = fma(y, fma(-b, y, np.ones_like(b)), y)
        keep = above | (part != 0x7FFFFF)
        np.testing.assert_array_equal(y[keep], ((np.float64(1) / b.astype(np.float64)).astype(f32))[keep])


def test_all_ones_divisor():
    """Every numerator significand over the divisor that the reciprocal's
    rounding is most sensitive to."""
    b = np.full(1, 0x3FFFFFFF, np.int32).view(f32)
    y = neighbour(b, True)
    y = fma(y, fma(-b, y, np.ones_like(b)), y)
    for part in np.array_split(np.arange(1 << 23, dtype=np.int32), 8):
        a = (part | 0x3F800000).view(f32)
        B, Y = np.broadcast_to(b, a.shape), np.broadcast_to(y, a.shape)
        np.testing.assert_array_equal(quotient(a, B, Y), a / B)


@pytest.mark.parametrize("above", [False, True])
def test_fast_quotient_to_its_lower_limit(above):
    """IEEE from |a| = 2^-102 up (a normal quotient); below, within an ulp."""
    rng = np.random.default_rng(200 + above)
    n = 300_000
    b = np.exp2(rng.uniform(-14, 20, n)).astype(f32)
    b[::8] = (b[::8].view(np.int32) | 0x7FFFFF).view(f32)   # all-ones significands
    y = neighbour(b, above)
    y[::8] = neighbour(b[::8], True)
    y = fma(y, fma(-b, y, np.ones_like(b)), y)
    sign = rng.choice([-1.0, 1.0], n)
    a = (sign * np.exp2(rng.uniform(-102, -39, n))).astype(f32)
    a[:64] = f32(2.0) ** -102
    np.testing.assert_array_equal(quotient(a, b, y), a / b)
    a = (sign * np.exp2(rng.uniform(-126, -102, n))).astype(f32)
    a[:64] = 0
    with np.errstate(all="ignore"):
        want, got = a / b, quotient(a, b, y)
    ulp = np.spacing(np.maximum(np.abs(want), np.finfo(f32).tiny))
    assert (np.abs(got.astype(np.float64) - want.astype(np.float64)) <= ulp).all()
    assert (got[:64] == 0).all()
