"""The integer-pipe product of the momentum kernels
(curvib_old_gb300/csrc/intmul.cuh), restated here on integers and checked
against the FP64 multiply bit for bit: significands at the edges of the
rounding (ties, all ones, one bit), exponents at both ends of its range, and
zeros of both signs."""
import random
import struct

M32 = 0xFFFFFFFF


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def value(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def split(x, shift):
    b = bits(x)
    h, l = b >> 32, b & M32
    m = 0 if ((h & 0x7FFFFFFF) | l) == 0 else (h & 0xFFFFF) | 0x100000
    s = ((m << 32 | l) << shift) & (2**64 - 1) if m else 0
    return s & M32, s >> 32, h & 0xFFF00000


def in_range(x):
    h = bits(x) >> 32
    return x == 0.0 or (((h & 0x7FFFFFFF) - (513 << 20)) & M32) < 1022 << 20


def int_mul(x, y):
    (al, ah, ase), (bl, bh, bse) = split(x, 5), split(y, 6)
    t = al * bl
    u = ah * bl + (t >> 32)
    v = al * bh + u
    assert u < 2**64 and v < 2**64
    w = ah * bh + (v >> 32)
    r, wl, wh = (v & M32) | ((t & M32) >> 11), w & M32, w >> 32
    top = wh & 0x100000
    if not top:
        wh, wl, r = (wh << 1 | wl >> 31) & M32, (wl << 1 | r >> 31) & M32, r << 1 & M32
    carry = (r + 0x7FFFFFFF + (wl & 1)) >> 32
    lo = wl + carry
    hi = (wh + (lo >> 32)) & M32
    lo &= M32
    if hi == 0:
        return value(((ase ^ bse) & 0x80000000) << 32 | lo)
    return value(((hi + ase + bse + top - (1024 << 20)) & M32) << 32 | lo)


def significands(rng):
    yield from (0, 1, 2, 3, 2**52 - 1, 2**52 - 2, 2**51, 2**51 + 1, 2**26, 2**26 + 1, 2**27 - 1, 0x5555555555555)
    for _ in range(60):
        b = rng.getrandbits(52)
        yield b
        yield b & ~((1 << rng.randrange(52)) - 1)  # few bits set: exact products and ties
        yield b | ((1 << rng.randrange(52)) - 1)


def test_product_is_the_rounded_one():
    rng = random.Random(1)
    ms = list(significands(rng))
    ends = (513, 514, 1022, 1023, 1024, 1533, 1534)
    for p in ms:
        for q in ms:
            x = value(rng.getrandbits(1) << 63 | rng.choice(ends) << 52 | p)
            y = value(rng.getrandbits(1) << 63 | rng.choice(ends) << 52 | q)
            assert in_range(x) and in_range(y)
            assert bits(int_mul(x, y)) == bits(x * y), (x, y)
    for z in (0.0, -0.0):
        for x in (1.5, -2.0**-510, 2.0**511, 0.0, -0.0):
            assert bits(int_mul(z, x)) == bits(z * x) and bits(int_mul(x, z)) == bits(x * z)


def test_range():
    assert all(in_range(x) for x in (0.0, -0.0, 2.0**-510, -(2.0**511), 1.9 * 2.0**511))
    assert not any(in_range(x) for x in (2.0**-511, 5e-324, 2.0**512, float("inf"), float("-inf"), float("nan")))


def int_triple(x):
    b = bits(x)
    e = b >> 52 & 0x7FF
    if not 1 <= e <= 2044:
        return x if b << 1 & (2**64 - 1) == 0 else 3.0 * x
    t = 3 * (b & (2**52 - 1) | 2**52)
    s = 2 if t >> 54 else 1
    r = (t + (s - 1) + (t >> s & 1)) >> s
    return value(((b & 2**63) + r + ((e + s - 1) << 52)) & (2**64 - 1))


def test_triple_is_the_rounded_one():
    rng = random.Random(2)
    for p in significands(rng):
        for e in (0, 1, 2, 1023, 2043, 2044, 2045, 2046):
            for sign in (0, 1):
                x = value(sign << 63 | e << 52 | p)
                assert bits(int_triple(x)) == bits(3.0 * x), x


def rounded(q):
    """A rational rounded to the nearest double, ties to even."""
    return q.numerator / q.denominator  # Python's integer division rounds correctly


def fma(a, b, c):
    from fractions import Fraction
    return rounded(Fraction(a) * Fraction(b) + Fraction(c))


def test_quotient_is_the_rounded_one():
    """quot_known: the quotient by a known divisor through its rounded reciprocal."""
    rng = random.Random(3)
    ms = list(significands(rng))
    for p in ms:
        for q in rng.sample(ms, 40):
            x = value(rng.getrandbits(1) << 63 | rng.choice((623, 1000, 1023, 1422)) << 52 | p)
            y = value(rng.getrandbits(1) << 63 | rng.choice((513, 1023, 1534)) << 52 | q)
            rcp = 1.0 / y
            r = x * rcp
            r = fma(fma(-y, r, x), rcp, r)
            r = fma(fma(-y, r, x), rcp, r)
            assert bits(r) == bits(x / y), (x, y)


def test_quotient_by_three_halves_is_the_rounded_one():
    """The projection's division by 1.5: one correction."""
    rng = random.Random(4)
    ms = list(significands(rng)) + [rng.getrandbits(52) for _ in range(20000)]
    for p in ms:
        x = value(rng.getrandbits(1) << 63 | rng.choice((623, 1022, 1023, 1422)) << 52 | p)
        r = x * (2.0 / 3.0)
        assert bits(fma(fma(-1.5, r, x), 2.0 / 3.0, r)) == bits(x / 1.5), x


def widen(u):
    """The double, or None where the kernel leaves the value to the conversion."""
    m = u & 0x7FFFFFFF
    if (m - 0x00800000) & M32 >= 0x7F000000 and m:
        return None
    h = (((u - (u >> 31 << 32)) >> 3) & 0x8FFFFFFF) + (896 << 20)
    return value((h if m else u) << 32 | (u << 29 & M32))


def narrow(v):
    """The FP32 bits, or None where the kernel leaves the value to the conversion."""
    b = bits(v)
    h, l = b >> 32, b & M32
    e = h >> 20 & 0x7FF
    if (e - 897) & M32 < 253:
        m = ((h & 0x7FFFFFFF) << 3 & M32 | l >> 29) - (896 << 23) & M32
        rest = l << 3 & M32
        return (h & 0x80000000) | (m + (rest > 0x80000000 or (rest == 0x80000000 and m & 1)))
    return h if (h & 0x7FFFFFFF) | l == 0 else None


def test_conversions_are_the_rounded_ones():
    import numpy as np
    rng = random.Random(5)
    for p in list(significands(rng)) + [rng.getrandbits(24) << 28 for _ in range(200)]:
        for e in (0, 1, 896, 897, 898, 1022, 1023, 1149, 1150, 1151, 2047):
            for sign in (0, 1):
                v = value(sign << 63 | e << 52 | p)
                n = narrow(v)
                assert (n is not None) == (897 <= e <= 1149 or v == 0.0)
                if n is not None:
                    assert n == int(np.float32(v).view(np.uint32)), v
    for u in [rng.getrandbits(32) for _ in range(20000)] + [0, 1 << 31, 1 << 23, 0x7F7FFFFF, 0x807FFFFF, 1]:
        f = float(np.uint32(u).view(np.float32))
        if 0 < u & 0x7FFFFFFF < 0x00800000 or u & 0x7FFFFFFF >= 0x7F800000:
            assert widen(u) is None, u
        else:
            assert bits(widen(u)) == bits(f), u


def test_ninefold_is_the_rounded_one():
    rng = random.Random(6)
    for p in list(significands(rng)) + [rng.getrandbits(52) for _ in range(5000)]:
        for e in (0, 1, 2, 1023, 2041, 2042, 2043, 2046):
            x = value(rng.getrandbits(1) << 63 | e << 52 | p)
            b = bits(x)
            if not 1 <= e <= 2042:
                continue  # zeros as they are, the others by the multiply
            t = 9 * (b & (2**52 - 1) | 2**52)
            s = 4 if t >> 56 else 3
            r = (t + (1 << (s - 1)) - 1 + (t >> s & 1)) >> s
            assert bits(9.0 * x) == ((b & 2**63) + r + ((e + s - 1) << 52)) & (2**64 - 1), x
