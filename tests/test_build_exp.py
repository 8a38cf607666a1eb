"""CPU restatement of the kernel-matrix build's exponential exp(-E 2^e)
(csrc/iexp.cuh: iexp_parts_core) and of its level assembly with the offset left to
the row (assemble_w_bits), checked against exact arithmetic.  The tables are read
from the generated header.

Error budget of Z = exp(g) 2^62 before the final rounding, in 2^-64 of the value:
the product of the lower parts 4 (the table's 23 dropped bits times 2^-21) + 4 (the
polynomial's 13 dropped bits times 2^-10, centred), the square and the shift 1, the
tables 2 + 1, the last product 4, the cubic term 0.5, and m ln2 m / 2."""
import os
import random
import re

import pytest

mp = pytest.importorskip("mpmath")
mp.mp.dps = 50
M64 = (1 << 64) - 1
HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "ferebus-v7_gb300", "csrc", "iexp_table.h")


def _table(name):
    with open(HEADER) as f:
        s = f.read()
    s = s[s.index(name):]
    return [int(v, 16) for v in re.findall(r"0x([0-9a-f]+)ULL", s[s.index("{"):s.index("}")])]


def _define(name):
    with open(HEADER) as f:
        return int(re.search(rf"#define {name} 0x([0-9a-f]+)", f.read()).group(1), 16)


TAB, FINE = _table("g_iexp_tab1024"), _table("g_iexp_fine1024")
LN2, L2E32 = _define("IEXP_LN2"), _define("IEXP_L2E32")


def _parts(E, F):
    """iexp_common_parts: (Z, m, table index)."""
    top = (1 << 32) - 1 if F >= 45 else (1 << (F - 13)) - 1
    E = min(E >> 32, top) << 32 | (E & 0xFFFFFFFF)
    frac = (E << (64 - F)) & M64 if F <= 64 else E >> (F - 64)
    x13 = E >> min(F - 13, 63)
    assert x13 < 1 << 32
    m = ((x13 * L2E32 >> 32) + 2 + (1 << 12)) >> 12
    g = (m * LN2 - frac) & M64
    j, k = g >> 54, (g >> 44) & 1023
    t = (g & ((1 << 44) - 1)) - (1 << 43)
    th = t >> 12
    assert -(1 << 31) <= th < 1 << 31
    eps = t + ((th * th) >> 41)
    a, b = FINE[k] >> 23, eps >> 13
    assert a < 1 << 31 and -(1 << 31) <= b < 1 << 31
    d = FINE[k] + eps + ((a * b) >> 28)
    assert 0 < d < 1 << 55
    Th, Tl, dh, dl = TAB[j] >> 32, TAB[j] & 0xFFFFFFFF, d >> 32, d & 0xFFFFFFFF
    mid = Th * dl + Tl * dh + (3 << 30)
    assert mid < 1 << 64
    return TAB[j] + Th * dh + (mid >> 32), m, j


@pytest.mark.parametrize("F", [20, 40, 45, 58, 64, 65, 90, 127])
def test_parts_within_the_error_budget(F):
    rnd = random.Random(F)
    for _ in range(4000):
        top = rnd.uniform(max(-64.0, -F), 6.4)   # x up to ~85, where the matrix's unit has long ended
        E = int(2.0 ** (top + F) * rnd.uniform(1.0, 2.0))
        if not 0 <= E < 1 << 62:
            continue
        Z, m, j = _parts(E, F)
        exact = mp.exp(-mp.mpf(E) * mp.mpf(2) ** -F)
        err = abs(mp.mpf(Z) * mp.mpf(2) ** (-62 - m) / exact - 1) * mp.mpf(2) ** 64
        assert err <= 17 + m / 2, (E, err, m)
        assert j <= 710 and 1 << 61 < Z < (1 << 63) + (1 << 52)


@pytest.mark.parametrize("F", [20, 43, 44, 45, 58, 64, 65, 127])
def test_zero_and_large_arguments(F):
    Z, m, _ = _parts(0, F)
    for e2 in (2, 4, 10):  # 1 in the matrix's unit, exactly
        assert ((Z >> (m + e2 - 1)) + 1) >> 1 == 1 << (62 - e2)
    for E in ((1 << 62) - 1, (1 << 61) + 12345):
        if E >> F >= 1100:
            _, m, _ = _parts(E, F)
            assert m >= 1100


def test_assembly_with_the_offset_left_to_the_row():
    bias_h = (1 << 22) * 0x0101010101 + 0x4B000000 * ((1 << 24) + (1 << 8) + 1)
    bias_lo = (1 << 22) * 0x010101 + 0x4B000000 * ((1 << 8) + 1)
    lim = 7 * 36 * (1 << 14)
    rnd = random.Random(3)
    for _ in range(2000):
        S = [rnd.randint(-lim, lim) for _ in range(8)]
        b = [0x4B400000 + v for v in S]
        p = [(b[i] * 256 + b[i + 1]) & 0xFFFFFFFF for i in (0, 2, 5)]
        for u in range(53, 61):
            H = ((p[0] << 24) + (p[1] << 8) + b[4]) & M64
            Lo = (p[2] << 8) + b[7]
            W = ((H << (u - 48)) + ((Lo + (1 << (71 - u)) - bias_lo) >> (72 - u)) - (bias_h << (u - 48))) & M64
            ref = (sum(S[L] << (32 - 8 * L) for L in range(5)) << (u - 48)) + \
                (((S[5] << 16) + (S[6] << 8) + S[7] + (1 << (71 - u))) >> (72 - u))
            assert W == ref & M64, (S, u)
