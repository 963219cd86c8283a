"""The arithmetic of the exact slice sums (csrc/phk_fixed.cuh), restated on the
host: which values the digits hold, that they hold them exactly, and that the
counters' bounds between two carries hold.

FP64: w 2^(e - base) as three unsigned 19-bit digits and the signed rest, base <=
e <= base + 21, bits below the unit returned (add_digits, add_outside).  FP32:
three digits by adding and subtracting 1.5 2^23 units (FixHist32)."""
from fractions import Fraction

import numpy as np
import pytest

M = (1 << 19) - 1
VALUES = 8190           # between two carries
WINDOW = 21


def _split64(u, base):
    """(digits or None, what is left)."""
    bits = int(np.float64(u).view(np.uint64))
    e = (bits >> 52) & 0x7ff
    w = (bits & ((1 << 52) - 1)) | (1 << 52)
    if bits >> 63:
        w = -w
    s = e - base
    if 0 <= s <= WINDOW:
        v, left = w << s, 0.0
    elif 1 <= -s <= 52:
        v = -(-w >> -s) if w < 0 else w >> -s
        top = np.uint64(bits & ~((1 << -s) - 1)).view(np.float64)
        left = float(u) - float(top)
    else:
        return None, float(u)
    return (v & M, (v >> 19) & M, (v >> 38) & M, v >> 57), left


@pytest.mark.parametrize('base', [1005 - 18, 82, 1982])
def test_fp64_digits_are_exact(base):
    rs = np.random.RandomState(1)
    u = rs.choice([-1., 1.], 4000) * np.ldexp(
        rs.uniform(1, 2, 4000), rs.randint(base - 80, base + 30, 4000) - 1023)
    u[:4] = [np.ldexp(2 - 2.0**-52, base + WINDOW - 1023),
             -np.ldexp(2 - 2.0**-52, base + WINDOW - 1023),
             np.ldexp(1., base - 1023), -np.ldexp(1., base - 1023 - 52)]
    unit = Fraction(2) ** (base - 1075)
    for x in u:
        d, left = _split64(x, base)
        if d is None:
            assert left == x
            continue
        assert all(0 <= q <= M for q in d[:3])
        total = d[0] + (d[1] << 19) + (d[2] << 38) + (d[3] << 57)
        assert total * unit + Fraction(left) == Fraction(float(x))
        assert abs(Fraction(left)) < unit
        assert -(1 << 17) <= d[3] < (1 << 17)


def test_fp64_counters_stay_in_range():
    # a carried digit, and VALUES more of the largest
    assert M + VALUES * M < 1 << 32
    assert (1 << 29) + VALUES * (1 << 17) + (1 << 13) < 1 << 31


def _value(d, base):
    """digits_value: d as 32-bit counters (the last signed)."""
    U = (1 << 64) - 1
    h, l = (d[3] << 19) + d[2], (d[1] << 19) + d[0]
    lo = ((h << 38) & U) + l & U
    hi = (h >> 26) + (lo < l) & U
    if not hi | lo:
        return 0.
    neg = hi >> 63
    if neg:
        lo = -lo & U
        hi = (~hi & U) + (lo == 0) & U
    lz = 128 - ((hi << 64) | lo).bit_length()
    top = (hi << lz & U) | lo >> (64 - lz) if hi else lo << (lz - 64)
    below = int(bool(hi) and (lo << lz & U) != 0)
    r = top >> 11
    r += ((top & 0x7ff) << 1 | below) + (r & 1) > 0x800
    r += 74 - lz + base << 52
    return float(np.uint64(r | neg << 63).view(np.float64))


@pytest.mark.parametrize('base', [82, 1005, 1900])
def test_fp64_value_is_rounded_once(base):
    rs = np.random.RandomState(3)
    unit = Fraction(2) ** (base - 1075)
    for n in range(6000):
        k = rs.randint(1, 33)
        d = [int(rs.randint(0, 1 << k, dtype=np.int64)) for _ in range(3)]
        d.append(int(rs.randint(-(1 << k - 1), 1 << k - 1, dtype=np.int64))
                 if n % 3 else -(n % 2))
        if n % 5 == 0:       # ties: 53 bits and a half
            d = [1 << 19 + n % 4, 0, 0, 0] if n % 2 else \
                [0, 0, 1 << 15, 1 << 12 + n % 3]
            d[0] += n % 3
        if n == 0:
            d = [0, 0, 0, 0]
        total = d[0] + (d[1] << 19) + (d[2] << 38) + (d[3] << 57)
        # Python rounds the quotient of two integers once
        q = Fraction(total) * unit
        assert _value(d, base) == q.numerator / q.denominator, d


@pytest.mark.parametrize('e', [-106, -10, 0, 100])
def test_fp32_digits_are_exact(e):
    f = np.float32
    rs = np.random.RandomState(2)
    top = f(np.ldexp(1.5, e + 17))
    mid, low = f(top * f(2.0**-18)), f(top * f(2.0**-36))
    lo, hi = max(e - 26, -148), min(e + 14, 127)
    u = (rs.choice([-1., 1.], 100000) *
         2.0**rs.uniform(lo, hi, 100000)).astype(f)
    with np.errstate(over='ignore', invalid='ignore'):
        h = f(u + top)
        r = f(u - f(h - top))
        m = f(r + mid)
        q = f(r - f(m - mid))
        l = f(q + low)
        ok = (np.abs(u) < f(top * f(1 / 128.))) & (f(l - low) == q)
    d = [v.view(np.int32).astype(np.int64) - int(c.view(np.int32))
         for v, c in ((h, top), (m, mid), (l, low))]
    unit = Fraction(2) ** (e - 42)
    for i in np.flatnonzero(ok)[::41]:
        total = (int(d[0][i]) << 36) + (int(d[1][i]) << 18) + int(d[2][i])
        assert total * unit == Fraction(float(u[i]))
    assert np.max(np.abs(d[0][ok])) <= 1 << 17
    assert max(np.max(np.abs(d[k][ok])) for k in (1, 2)) <= 1 << 17
    # the window: 2^-19 to 2^10 of the typical value at least
    a = np.abs(u.astype(np.float64))
    inside = (a >= np.ldexp(1., max(e - 19, -126))) & (a < np.ldexp(1., e + 10))
    assert np.all(ok[inside])
    # counters: a carried digit and as many more of the largest
    values = 16380
    assert (1 << 18) + values * (1 << 17) < 1 << 31
    assert (1 << 29) + values * 98304 + (1 << 15) < 1 << 31
