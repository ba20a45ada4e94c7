"""The even/odd Montgomery rows (csrc/field.cuh eo_*) restated on 32-bit words:
every carry that the device code drops must be zero for the operand ranges it
states, and the results must stay below the bounds that the lazy callers rely
on.  The x-only doubling chain and the quotient estimate of the MSM's last
reduction step (csrc/curve.cuh sl_dbl_many, qlin) are checked the same way."""
import random

import pytest

FR = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
FQ = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47
M32 = (1 << 32) - 1


def words(x):
    return [(x >> (32 * i)) & M32 for i in range(8)]


def value(w):
    return sum(x << (32 * i) for i, x in enumerate(w))


def mad(acc, ws, b, carry=0):
    """The chain of four lo/hi multiply-adds over an eight-word accumulator: (words, carry out)."""
    t = value(acc) + carry + sum(x * b << (64 * i) for i, x in enumerate(ws))
    return words(t), t >> 256


def redc(e, o, p):
    n0 = -pow(p, -1, 1 << 32) % (1 << 32)
    m = e[0] * n0 & M32
    pw = words(p)
    o, c = mad(o, pw[1::2], m)
    assert c == 0
    e, c = mad(e, pw[0::2], m)
    assert e[0] == 0
    o = words(value(o) + (c << 224))
    return e, o


def mad_shift(e, o, aw, b):
    t = o[0] + e[1]
    o = [t & M32] + o[1:]
    n, c = mad(e[2:] + [0, 0], aw[1::2], b, t >> 32)
    assert c == 0
    o, c = mad(o, aw[0::2], b)
    assert n[7] + c <= M32, "carry out of the ninth word"
    n[7] += c
    return o, n


def mad_plain(e, o, cw, d):
    o, c = mad(o, cw[1::2], d)
    assert c == 0
    e, c = mad(e, cw[0::2], d)
    assert o[7] + c <= M32
    o[7] += c
    return e, o


def product(pairs, p):
    """sum of a b over one or two pairs, divided by 2^256 modulo p."""
    e, o = [0] * 8, [0] * 8
    for i in range(8):
        for k, (a, b) in enumerate(pairs):
            aw, bw = words(a), words(b)
            if i and not k:
                e, o = mad_shift(e, o, aw, bw[i])
            else:
                e, o = mad_plain(e, o, aw, bw[i])
        e, o = redc(e, o, p)
    r = value(o) + (value(e) >> 32)
    assert r < 1 << 256
    return r


@pytest.mark.parametrize("p", [FR, FQ], ids=["fr", "fq"])
def test_rows_and_bounds(p):
    rng = random.Random(p & 0xFFFF)
    rinv = pow(1 << 256, -1, p)
    edges = [0, 1, p - 1, p, 2 * p - 1, 2 * p, (1 << 224) - 1, 1 << 253, (1 << 254) - 1]
    cases = [(x, y) for x in edges for y in edges]
    cases += [(rng.randrange(2 * p), rng.randrange(2 * p)) for _ in range(400)]
    for a, b in cases:
        r = product([(a, b)], p)
        assert r % p == a * b * rinv % p and r * 100 < 176 * p
        r = product([(a, b), (b, a)], p)
        assert r % p == 2 * a * b * rinv % p and r * 100 < 252 * p
    # one factor may be any 256-bit value, the other must leave room for p
    big = (1 << 256) - 1
    for a in (p - 1, 2 * p - 1, 4 * p, (1 << 256) - 1 - p):
        for b in (big, big ^ M32, rng.randrange(1 << 256)):
            e, o = [0] * 8, [0] * 8
            for i in range(8):
                e, o = mad_shift(e, o, words(a), words(b)[i]) if i else mad_plain(e, o, words(a), words(b)[0])
                e, o = redc(e, o, p)
            assert (value(o) + (value(e) >> 32)) % p == a * b * rinv % p


def test_x_only_doublings():
    def dbl(pt):
        x, y = pt
        s = 3 * x * x * pow(2 * y, -1, FQ) % FQ
        x3 = (s * s - 2 * x) % FQ
        return x3, (s * (x - x3) - y) % FQ

    rng = random.Random(7)
    for m in (1, 2, 3, 15, 127):
        pt = (1, 2)
        for _ in range(rng.randrange(1, 6)):
            pt = dbl(pt)
        z = rng.randrange(1, FQ)
        x, y, zz, zzz = pt[0] * z * z % FQ, pt[1] * z ** 3 % FQ, z * z % FQ, z ** 3 % FQ
        X, Z, yn, yd, M, C, D = x, zz, y, zzz, 1, 1, 1
        for i in range(m + 1):
            X2, Z2, XZ, CC, CD, DD = X * X, Z * Z, X * Z, C * C, C * D, D * D
            A, B, C, D, yn, yd = X2 * X2, XZ * Z2, XZ * X2, Z2 * Z2, yn * M, yd * (Z2 if i else 1)
            A, B, C, D, yn, yd = (v % FQ for v in (A, B, C, D, yn, yd))
            if i:
                M = (2 * CC + 120 * CD - 144 * DD) % FQ
            if i < m:
                X, Z = (A - 24 * B) % FQ, (4 * C + 12 * D) % FQ
        yn = yn * M % FQ
        t = Z * yd % FQ
        ZZ, ZZZ, X3, Y3 = t * t, t ** 3, X * yd * t, yn * Z * t * t
        want = pt
        for _ in range(m):
            want = dbl(want)
        assert X3 * pow(ZZ, -1, FQ) % FQ == want[0] and Y3 * pow(ZZZ, -1, FQ) % FQ == want[1]


def test_quotient_estimate():
    c = (1 << 280) // FQ
    assert c == 88753990
    rng = random.Random(3)
    top = 266 * 2 * FQ
    for t in [0, 1, FQ - 1, FQ, top] + [k * FQ + d for k in range(0, 533, 7) for d in (-1, 0, 1) if k] + \
            [rng.randrange(top) for _ in range(2000)]:
        q = ((t >> 248) * c) >> 32
        assert 0 <= t - q * FQ < 11 * FQ // 10


def test_reduction_passes():
    """The reduction's passes cover every width: all bits folded once, each pass's first step within 320 threads."""
    for c in range(4, 23):
        arrays, left, passes = 1, c - 1, 0
        while left:
            m = min(left, 9)
            while m > 1 and arrays << (m - 1) > 320:
                m -= 1
            assert arrays << (m - 1) <= 320 and 128 * ((arrays + 1) << (m - 1)) <= 1 << 16
            arrays, left, passes = arrays + m, left - m, passes + 1
        assert arrays == c and passes <= 6
