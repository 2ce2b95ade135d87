"""The seven-digit scheme of oz8_common.cuh, restated on the CPU.

The FP64-accurate kernels (oz_xc64.cu, oz_gram64.cu) cut a value into 55
fraction bits below its group's power of two, these into seven balanced 8-bit
digits, sum the digit products of a level exactly, recombine the eight level
sums into one 64-bit integer T and round T 2^base to FP64.  Restated here with
Python integers and numpy FP32 / uint operations, instruction for instruction
where the width of a register matters:
  * the digits reproduce the truncated value, and lie in their ranges;
  * T is the exact sum to its stated unit and fits 63 bits, at the extremes of
    every kernel's group length and stacking of slices;
  * the fast conversion equals the general one wherever a kernel uses it.
"""
import math
import random
from fractions import Fraction

import numpy as np
import pytest

f32 = np.float32
S = 7
BASE = 2099
M63 = (1 << 63) - 1


def bits(v):
    return int(np.float64(v).view(np.uint64))


def bexp(v):
    return (bits(v) >> 52) & 0x7FF


def fixed(v, E):
    """|v| truncated to 55 fraction bits below 2^(E - 1022) (oz8_fixed)."""
    b = bits(v)
    m = ((b & 0xFFFFFFFFFFFFF) | 1 << 52) << 2
    # the 32-bit subtraction: es - (hi without its sign) with es all ones below E
    sh = min((((((E << 20) | 0xFFFFF) if E else 0xFFFFFFFF) - ((b >> 32) & 0x7FFFFFFF)) & 0xFFFFFFFF) >> 20, 63)
    return m >> sh


def digits(v, E):
    """The digits of |v|, from the bytes of oz8_fixed plus 0x80 in six of them."""
    u = fixed(v, E) + 0x808080808080
    return [u >> 48] + [((u >> (40 - 8 * t)) & 0xFF) - 128 for t in range(6)]


def signed(v, E):
    s = -1 if bits(v) >> 63 else 1
    return [s * d for d in digits(v, E)]


def combine(lev, half):
    """oz8_combine on integer level sums; `half`: groups of 256 rows drop a bit.
    Returns the 64-bit register and the same without wrapping."""
    a0, a1 = lev[0] * 256 + lev[1], lev[2] * 256 + lev[3]

    def even(x):  # adding 1.5 2^24 in FP32 to an integer up to 2^23 (and the carry of a level): units of 2
        assert abs(x) <= (1 << 23) + 256
        y = int(f32(f32(x) + f32(25165824.0)))
        assert y < 1 << 25  # beyond it the spacing is 4
        return (y - 25165824) // 2

    y4 = even(lev[4])
    f5 = (lev[4] - 2 * y4) * 256 + lev[5]
    y5 = even(f5)
    f6 = (f5 - 2 * y5) * 256 + lev[6]
    a6 = even(f6) * 256 + even(lev[7]) + 8192
    assert max(abs(a0), abs(a1), abs(a6)) < 1 << 31
    t = a1 * 131072 + y4 * 1024 + y5 * 4 + (a6 >> 14)
    T = ((t + ((t >> 1) & 1)) >> 1) + (a0 << 32) if half else t + (a0 << 33)
    w = T & ((1 << 64) - 1)
    return (w - (1 << 64) if w >> 63 else w), T


def scaled(T, base):
    """oz8_scaled: nearest, ties away; 0 below the normal range, infinity above."""
    if T == 0:
        return 0.0
    A = abs(T)
    lz = 64 - A.bit_length()
    m = ((A << (lz - 1)) + 0x200) >> 10
    e = 1085 - lz + base
    b = m + ((e & 0xFFFFFFFF) << 52) & ((1 << 64) - 1)
    if not 0 <= e < 2046:
        b = 0x7FF << 52 if e > 0 else 0
    return float(np.uint64(b | (1 << 63 if T < 0 else 0)).view(np.float64))


def scaled_fast(T, base):
    """oz8_scaled_fast, with its 32-bit registers."""
    sg = -1 if T < 0 else 0
    A = ((T ^ sg) - sg) & ((1 << 64) - 1)
    ah, al = A >> 32, A & 0xFFFFFFFF
    p = ah.bit_length() - 1
    ls = (30 - p) & 31
    hi = (((ah << 32 | al) << ls) >> 32) & 0xFFFFFFFF
    m = ((hi << 32 | (al << ls) & 0xFFFFFFFF) + 0x200) >> 10
    rh = ((m >> 32) + ((p + base + 1054) & 0xFFFFFFFF) * 0x100000) & 0xFFFFFFFF
    return float(np.uint64((rh | (sg & 0x80000000)) << 32 | m & 0xFFFFFFFF).view(np.float64))


def value(v, E):
    """The value the digits stand for, in units of 2^(E - 1022)."""
    return sum(Fraction(d, 1 << (7 + 8 * t)) for t, d in enumerate(signed(v, E)))


@pytest.mark.parametrize("E", [1023, 300, 1700])
def test_digits_reproduce_the_truncated_value(E):
    rng = random.Random(E)
    vals = [math.ldexp(rng.uniform(0.5, 1.0), E - 1022 - rng.choice([0, 0, 1, 2, 3, 9, 30, 54, 60])) for _ in range(300)]
    vals += [math.ldexp(1 - 2.0 ** -53, E - 1022), math.ldexp(0.5, E - 1022), 0.0,
             math.ldexp(0.99609375, E - 1022), math.ldexp(0.99609374999999, E - 1022)]
    for v in vals:
        for x in (v, -v):
            d = digits(x, E)
            assert 0 <= d[0] <= 128 and all(-128 <= t <= 127 for t in d[1:])
            exact = Fraction(x) / Fraction(2) ** (E - 1022)
            err = abs(exact) - abs(value(x, E))
            assert 0 <= err < Fraction(1, 1 << 55)
            if abs(exact) >= Fraction(1, 8):
                assert err == 0


def _row_blocks(dx, dy, F, rows):
    """The level sums of each row block q (weight 2^(-8 q)) for `rows` rows of
    constant columns with digits dx, dy: TMEM column c of row block q holds the
    pairs (slice t = F a + q of Y, slice u of X) with c = F a + u."""
    for q in range(min(F, S)):
        lev = [0] * 8
        for t in range(q, S, F):
            for u in range(S):
                c = t - q + u
                if c < 8:
                    lev[c] += dy[t] * dx[u] * rows
        yield q, lev


def _constants():
    yield 1 - 2.0 ** -53
    yield 0.997
    yield 1 - 1e-12
    yield 0.99609375  # a top digit rounded up to 128
    rng = random.Random(5)
    for _ in range(60):
        yield rng.uniform(0.9962, 1.0)
    for _ in range(30):
        yield rng.uniform(0.5, 1.0)


# (slices stacked, rows of a group): the three variants of the Gram kernel
@pytest.mark.parametrize("F,rows", [(2, 128), (4, 256), (8, 256)])
def test_gram_groups_fit_63_bits(F, rows):
    """Columns of constants just below a power of two: the largest sums a group
    can hold.  (T of 256-row groups once took 64 bits: their entries came back
    with the opposite sign.)"""
    half = rows == 256
    E = 1022
    cs = list(_constants())
    for x in cs[:6]:
        for y in cs:
            for sx, sy in ((1, 1), (1, -1), (-1, -1)):
                dx, dy = signed(sx * x, E), signed(sy * y, E)
                got = Fraction(0)
                for q, lev in _row_blocks(dx, dy, F, rows):
                    reg, T = combine(lev, half)
                    assert reg == T and abs(T) <= M63, (x, y, F)
                    unit = Fraction(1, 1 << (54 if half else 55)) / (1 << 8 * q)
                    got += T * unit
                want = rows * value(sx * x, E) * value(sy * y, E)
                # products of levels >= 8 left out; T rounded to its unit in every row block
                assert abs(got - want) <= Fraction(rows * 6, 1 << 64) + Fraction(3, 1 << 55)


def test_update_rows_fit_63_bits():
    """64 columns of the update: T within 2^62 and a bit."""
    E = 1022
    for x in (1 - 2.0 ** -53, 0.997, 0.99609375):
        for y in _constants():
            dx, dy = signed(x, E), signed(-y, E)
            lev = [64 * sum(dx[t] * dy[L - t] for t in range(S) if 0 <= L - t < S) for L in range(8)]
            reg, T = combine(lev, False)
            assert reg == T and abs(T) < 1 << 62
            want = 64 * value(x, E) * value(-y, E)
            assert abs(Fraction(T, 1 << 55) - want) <= Fraction(64 * 6, 1 << 64) + Fraction(1, 1 << 55)


def test_fast_conversion_where_it_is_used():
    """The sums of exponents that oz8_ordinary lets pass: the fast conversion is
    the general one, and both are the nearest FP64 number (ties away from zero);
    with the weight 2^-56 of a Gram's last row block too.  Far below, where two
    scales are usable and their product is not, it would not be."""
    rng = random.Random(9)
    Ts = [1 << 32, (1 << 32) + 1, (1 << 62) + 5, (1 << 63) - 1, (1 << 54) + (1 << 1), (1 << 53) - 1]
    Ts += [rng.getrandbits(b) | 1 << (b - 1) for b in range(33, 64) for _ in range(6)]
    for e2 in (1120, 1121, 1500, 2046, 2900, 3019, 3020):
        for shift in (0, 56):
            for T in Ts + [-t for t in Ts]:
                base = e2 - BASE - shift
                y = scaled(T, base)
                assert scaled_fast(T, base) == y and math.isfinite(y)
                err = abs(Fraction(y) - Fraction(T) * Fraction(2) ** base)
                assert err <= Fraction(2) ** (base + max(T.bit_length() - 54, -1))
                assert err == 0 or T.bit_length() > 53
    assert scaled_fast(1 << 56, 2 * 359 - BASE) != scaled(1 << 56, 2 * 359 - BASE)  # 1e-200 x 1e-200


def _update_entry(x, c):
    """One entry of the update from digits: the result, and whether the sums of the
    top digits let it stand (oz_xc64.cu)."""
    Ex, Ec = max(map(bexp, x)), max(map(bexp, c))
    dx, dc = [signed(v, Ex) for v in x], [signed(v, Ec) for v in c]
    lev = [sum(a[t] * b[L_ - t] for a, b in zip(dx, dc) for t in range(S) if 0 <= L_ - t < S) for L_ in range(8)]
    reg, T = combine(lev, False)
    assert reg == T
    N, N2 = sum(abs(d[0]) for d in dx), sum(abs(d[0]) for d in dc)
    D = sum(abs(a[0] * b[0]) for a, b in zip(dx, dc))
    m = sum(v != 0 for v in c)
    if m < 2:
        return scaled(T, Ex + Ec - BASE), False
    kappa = f32(0.503) + f32(32.01) / f32(m - 1)
    need = f32(kappa * f32(N)) + f32(f32(kappa * f32(N2)) + (f32(32.01) * f32(len(x)) + f32(5330)) / f32(m - 1))
    return scaled(T, Ex + Ec - BASE), D >= need


def test_update_entries_that_stand_keep_the_bound_of_multiply_adds():
    """m 2^-53 sum |x_i c_i|, m the nonzeros of c, whatever the values' sizes; and
    random ones do stand."""
    rng = random.Random(17)
    stood = dict.fromkeys(("even", "graded", "sparse", "top"), 0)
    for trial in range(1600):
        kind = list(stood)[trial % 4]
        h = rng.choice([2, 3, 8, 16, 32, 64])
        x, c = [rng.gauss(0, 1) for _ in range(h)], [rng.gauss(0, 1) for _ in range(h)]
        if kind == "graded":
            x = [v * 10.0 ** -rng.uniform(0, 18) for v in x]
            c = [v * 10.0 ** -rng.uniform(0, rng.choice([1, 18])) for v in c]
        elif kind == "sparse":
            c = [v if rng.random() < 0.3 else 0.0 for v in c]
            c[0] = c[0] or 1.0
        elif kind == "top":  # values just below the places where a top digit rounds
            x = [rng.choice([1 - 2.0 ** -53, 0.0039, 0.00390624, 0.0117, 2.0 ** -30]) for _ in x]
        y, ok = _update_entry(x, c)
        if not ok:
            continue
        stood[kind] += h >= 32
        exact = sum(Fraction(a) * Fraction(b) for a, b in zip(x, c))
        mag = sum(abs(Fraction(a) * Fraction(b)) for a, b in zip(x, c))
        m = sum(v != 0 for v in c)
        assert abs(Fraction(y) - exact) <= m * Fraction(1, 1 << 53) * mag, (kind, h, trial)
    assert stood["even"] > 100 and stood["graded"] > 0 and stood["sparse"] > 20


@pytest.mark.parametrize("half", [False, True])
def test_rounding_of_the_sums_does_not_drift(half):
    """T is the level sums' exact integer to half a unit, up as often as down: a
    rounding that favours one direction would add up over a Gram's groups."""
    rng = random.Random(6)
    errs = []
    for _ in range(4000):
        lev = [rng.randint(-(1 << 20), 1 << 20) for _ in range(4)] + [rng.randint(-(1 << 22), 1 << 22) for _ in range(4)]
        T = combine(lev, half)[1]
        errs.append(float(T - Fraction(sum(s * 256 ** (7 - i) for i, s in enumerate(lev)), 1 << (16 if half else 15))))
    assert max(map(abs, errs)) <= (0.8 if half else 0.52)
    assert abs(np.mean(errs)) <= 4 * np.std(errs) / len(errs) ** 0.5
