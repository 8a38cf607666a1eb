"""CPU model of the fixed-point arithmetic of the tensor-core mode (csrc/panel.cu,
csrc/tc_common.cuh): the reciprocal square root of the pivots, the 62-bit fixed
point of the kernel matrix, the substitution in 60-bit fixed point and the
digits of its results.

Bounds, derived before the first run: the reciprocal square root errs by
2^-59 from e / 2 and 2^-59 from 3 e^2 / 8 cut to that unit, 3 x 2^-62 from e (the
low words' product and two high words cut off), 5/16 e^3 < 2^-61 from the series
and y0 times that again, all relative: below 2^-57; each conversion rounds
once, so it is within half a unit.
"""
import math
import random
import struct
from fractions import Fraction

import numpy as np


def _bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def _double(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def rsqrt_fixed(D, ulps):
    """The device function; ``ulps`` perturbs the single-precision estimate."""
    hi, lo = D >> 32, D & 0xFFFFFFFF
    h1, l1 = (hi, lo) if hi else (lo, 0)
    z = 32 - h1.bit_length()
    E = (3 if hi else -29) - z
    r = E & 1
    A = ((h1 << 32) | l1) << z
    assert A >> 63 == 1 and A < 2 ** 64
    ah, al = A >> 32, A & 0xFFFFFFFF
    sh = -(E >> 1) - 1
    mf = np.uint32((ah >> 8) + ((126 + r) << 23)).view(np.float32)
    assert 1 <= mf <= 4
    y0 = np.uint32(int(np.float32(1.0 / math.sqrt(float(mf))).view(np.uint32)) + ulps).view(np.float32)
    Y = int(np.float32(y0 + np.float32(1.0)).view(np.uint32)) - 0x3F800000
    assert 2 ** 22 <= Y <= 2 ** 23
    q = (Y * Y) << 17
    assert q < 2 ** 64
    m = A if r else A >> 1
    mh, ml, qh, ql = m >> 32, m & 0xFFFFFFFF, q >> 32, q & 0xFFFFFFFF
    e = (1 << 61) - ((ml * qh) >> 32) - (mh * qh + ((mh * ql) >> 32))
    assert abs(e) < 2 ** 41
    eh = e >> 10
    assert abs(eh) < 2 ** 31
    e2 = (eh * eh) >> 32
    assert e2 * 3 < 2 ** 32
    c2 = (e2 * 3) >> 14
    prod = Y * (e >> 3) + Y * c2
    assert abs(prod) < 2 ** 63
    y = (((Y * 256 - 1) << 32) | 0xFFFFFFFF) + (prod >> 19)
    assert 0 <= y < 2 ** 63
    return y, sh


def test_rsqrt_fixed_within_its_bound():
    rng = random.Random(5)
    cases = [4, 5, 7, 2 ** 60 - 1, 2 ** 59, 2 ** 59 - 1, 2 ** 59 + 1, 2 ** 58, 2 ** 58 - 1]
    cases += [rng.getrandbits(rng.randint(3, 60)) | 4 for _ in range(4000)]
    for D in cases:
        for ulps in (-1, 0, 1):  # the estimate is within 2^-22.9
            y, sh = rsqrt_fixed(D, ulps)
            assert 0 <= sh <= 28 and 2 ** 62 <= y + 2 ** 5
            got = Fraction(y) * Fraction(2) ** (sh - 62)
            # relative error: got = (1 + t) / sqrt(d), t = (got^2 d - 1) / 2 to first order
            t = abs(float((got ** 2 * Fraction(D, 2 ** 60) - 1) / 2))
            assert t <= 2.0 ** -57, (D, ulps, t)


def wrap(v, bits=64):
    assert -(1 << (bits - 1)) <= v < 1 << (bits - 1), v
    return v


def split30(X):
    r = X + (1 << 29)
    hi = min(max(r >> 32, -(1 << 28)), (1 << 28) - 1)
    h = (hi << 2) | ((r >> 30) & 3)
    return h, wrap((X - (h << 30) + (1 << 31)) % (1 << 32) - (1 << 31), 32)


def scale_entry(T, y, sh):
    lim = 1 << (29 - sh)
    yh, yl = y >> 32, y & 0xFFFFFFFF
    th = min(max(T >> 32, -lim), lim - 1)
    u = wrap(((th << 32) | (T & 0xFFFFFFFF)) << (sh + 2))
    uh, ul = u >> 32, u & 0xFFFFFFFF
    X = wrap(uh * yh + ((ul * yh) >> 32) + ((uh * (yl >> 1)) >> 31))
    return split30(X)


def substitute(T, L, ys, shs):
    """One row through a 16 x 16 block: the device's fixed-point steps, with
    the 64-bit range of every sum checked."""
    out = []
    for k in range(16):
        S, M = T[k], 0
        for c in range(k):
            lh, ll = split30(L[k][c])
            xh, xl = out[c]
            S = wrap(S - xh * lh)
            M = wrap(M + xh * ll + xl * lh)
        h, low = scale_entry(wrap(S - (M >> 30)), ys[k], shs[k])
        assert abs(h) <= 2 ** 30 and -2 ** 29 <= low < 2 ** 29
        out.append((h, low))
    return [(h << 30) + low for h, low in out]


def test_scale_entry_clamps_what_a_semidefinite_matrix_cannot_have():
    """|x| < 1 is exact to a few units; beyond it the high half is that of +-1."""
    rng = random.Random(4)
    for _ in range(4000):
        y, sh = rsqrt_fixed(rng.getrandbits(rng.randint(3, 60)) | 4, 0)
        T = rng.choice([-1, 1]) * rng.randrange(1 << (60 - sh))
        h, low = scale_entry(T, y, sh)
        want = (T * y) >> (62 - sh)
        if abs(want) < 2 ** 60 - 2 ** 30:
            assert abs(want - ((h << 30) + low)) <= 3
        big = rng.choice([-1, 1]) * rng.randrange(1 << (60 - sh), 1 << 62)
        assert abs(scale_entry(big, y, sh)[0]) >= 2 ** 30 - 4


def test_substitution_in_fixed_point():
    """Against exact rational substitution on the same block.  Bound: column
    k's right-hand side is off by its rounding (2^-61), the dropped Xl Ll (at
    most 15 x 2^58 2^-120), the shift (2^-60) and the block's own rounding
    (15 x 2^-61 |x|); the division by L_kk scales that by 1 / L_kk, plus y's
    2^-57 relative and 3 x 2^-60: below 2^-56 (1 + 1 / min L_kk), amplified by
    the block's conditioning, which max |inv(L)| bounds."""
    rng = np.random.default_rng(9)
    for cond in (0.0, 2.0, 6.0, 9.0):
        A = rng.normal(size=(40, 24)) * np.exp(-cond * np.linspace(0, 1, 24))
        G = A @ A.T + 1e-9 * np.eye(40)
        G /= 1.01 * G.diagonal().max()
        Lf = np.linalg.cholesky(G)
        blk, row = Lf[:16, :16], Lf[20, :16]
        L = [[round(Fraction(float(v)) * 2 ** 60) for v in r] for r in blk]
        D = [round(Fraction(float(blk[j, j])) ** 2 * 2 ** 60) for j in range(16)]
        ys, shs = zip(*(rsqrt_fixed(d, 0) for d in D))
        T = [round(sum(Fraction(float(row[c])) * Fraction(float(blk[k, c])) for c in range(k + 1)) * 2 ** 60)
             for k in range(16)]
        got = substitute(T, L, ys, shs)
        inv = np.abs(np.linalg.inv(blk)).max()
        tol = 2.0 ** -56 * (1 + inv) * (1 + 16 * inv * np.abs(blk).max())
        for k in range(16):
            assert abs(got[k] / 2.0 ** 60 - row[k]) <= tol, (cond, k, got[k] / 2.0 ** 60 - row[k], tol)


def to_fixed62(x, e):
    b = _bits(x)
    E = (b >> 52) & 0x7FF
    M = (b & ((1 << 52) - 1)) | (1 << 52)
    sh = E - 1075 + 62 - e
    if sh > 9:
        F = (1 << 62) - 1
    elif E == 0 or sh <= -63:
        F = 0
    else:
        F = M << sh if sh >= 0 else (M + (1 << (-sh - 1))) >> (-sh)
    return -F if b >> 63 else F


def test_to_fixed62_rounds_once_and_saturates():
    rng = random.Random(6)
    for _ in range(20000):
        e = rng.randint(-40, 40)
        x = rng.choice([-1, 1]) * 2.0 ** (e - rng.expovariate(0.1)) * rng.uniform(0.5, 1.0)
        F = to_fixed62(x, e)
        assert abs(Fraction(x) * Fraction(2) ** (62 - e) - F) <= Fraction(1, 2)
        assert abs(F) < 2 ** 62
    assert to_fixed62(0.0, 3) == 0 and to_fixed62(5e-324, 0) == 0
    assert to_fixed62(math.nextafter(2.0 ** 5, 0), 5) == (2 ** 53 - 1) << 9
    top = 2 ** 62 - 1
    assert to_fixed62(2.0 ** 5, 5) == top and to_fixed62(-1e30, 5) == -top
    assert to_fixed62(math.inf, 9) == top and to_fixed62(-math.inf, 9) == -top


def fixed62_to_double(T):
    a = abs(T)
    lz = 64 - a.bit_length()
    if lz == 64:
        return 0.0
    a = (a << lz) & (2 ** 64 - 1)
    mant = (a >> 11) + ((a >> 10) & 1)
    r = ((1024 - lz) << 52) - (1 << 52) + mant
    return math.copysign(_double(r), T)


def test_fixed62_to_double_rounds_to_nearest():
    rng = random.Random(7)
    cases = [1, 2, 3, 2 ** 62 - 1, 2 ** 62, 2 ** 53 + 1, 2 ** 54 - 1, 2 ** 63 - 1]
    cases += [rng.getrandbits(rng.randint(1, 63)) | 1 for _ in range(20000)]
    for T in cases:
        for sgn in (1, -1):
            got = fixed62_to_double(sgn * T)
            want = Fraction(sgn * T, 2 ** 62)
            assert abs(Fraction(got) - want) <= Fraction(math.ulp(float(want))) / 2
    assert fixed62_to_double(0) == 0.0


def digits(X):
    """d_0 .. d_6 of X = x 2^60 as the kernel forms them: bytes of F + bias."""
    G = ((X + 16) >> 5) + 0x808080808080
    return [(G >> 48)] + [((G >> (8 * (6 - p))) & 0xFF) - 128 for p in range(1, 7)]


def test_digits_of_a_fixed_point_entry():
    rng = random.Random(8)
    cases = [0, 1, -1, 15, 16, -16, -17, 2 ** 60, -2 ** 60, 2 ** 60 - 1, 1 - 2 ** 60]
    cases += [rng.choice([-1, 1]) * rng.getrandbits(rng.randint(1, 60)) for _ in range(20000)]
    for X in cases:
        d = digits(X)
        F = sum(v << (8 * (6 - p)) for p, v in enumerate(d))
        assert abs(Fraction(X, 32) - F) <= Fraction(1, 2)
        assert all(-128 <= v <= 127 for v in d[1:]) and -128 <= d[0] <= 128
