"""The tensor-core products' present arithmetic restated in numpy (CPU): the balanced base-256 digits
of xs::fixed / xs::digit with the level sums of k_xs_gemm's epilogue (S = 6 and 7), and the four
BF16 slices of tc::slice4f with tc::join and tc::scaled.  Tolerances are the roundings each scheme
states; sums are compared with exact rational arithmetic."""
from fractions import Fraction

import numpy as np
import pytest

F32 = np.float32


def bits_of(S):
    return 8 * S - 1


def fixed(x, e, S):
    """round(|x| 2^(bits - e)) with x's sign, halves away from zero, as a Python int."""
    m, ex = np.frexp(abs(float(x)))
    n = int(m * 2.0 ** 53)                       # |x| = n 2^(ex - 53)
    sh = 53 - int(ex) - (bits_of(S) - e)         # right shift
    v = n << -sh if sh <= 0 else ((n >> (sh - 1)) + 1) >> 1
    return -v if x < 0 else v


def digits(v, S):
    """Balanced base-256 digits of v, leading one first: bytes of v plus 128 in every digit but the
    leading one (xs::digit)."""
    w = v + sum(128 << (8 * t) for t in range(S - 1))
    assert -(1 << 63) <= w < 1 << 63
    return [w >> (8 * (S - 1))] + [((w >> (8 * (S - 1 - j))) & 255) - 128 for j in range(1, S)]


def join(levels, S):
    """Level sums to FP64 as the epilogue does: 64-bit units of 2^-61, one rounding.  S = 7: the last of
    the seven accumulators holds levels 6 and 7, in single precision."""
    head = (levels[0] << 16) + (levels[1] << 8) + levels[2]
    assert abs(head) < 1 << 31                   # 32-bit integers
    v = (head << 31) + (levels[3] << 23) + (levels[4] << 15) + (levels[5] << 7)
    if S == 7:
        v += int(np.rint(F32(levels[6]) + F32(levels[7] / 256.0))) >> 1
    assert abs(v) < 1 << 63
    return float(Fraction(v, 1 << 61))           # Fraction -> float rounds to nearest


@pytest.mark.parametrize("S", [6, 7])
@pytest.mark.parametrize("e", [0, 3, -5])
def test_digits_restore_the_rounded_operand(S, e):
    rng = np.random.default_rng(S)
    top = 2.0 ** e
    below = np.nextafter(top, 0)
    xs = [0.0, top, -top, below, -below, 5e-324, -5e-324, 2.0 ** -1022, top * (1 + 2.0 ** -40), top / 3, -top / 256]
    xs += list(top * rng.uniform(-1, 1, 200)) + list(top * 2.0 ** rng.uniform(-70, 0, 200) * rng.choice([-1, 1], 200))
    for x in xs:
        v = fixed(x, e, S)
        d = digits(v, S)
        assert sum(q << (8 * (S - 1 - j)) for j, q in enumerate(d)) == v
        assert all(-128 <= q <= 127 for q in d[1:]) and abs(d[0]) <= 129
        unit = Fraction(2) ** (e - bits_of(S))
        assert abs(Fraction(x) - v * unit) <= unit / 2


@pytest.mark.parametrize("S", [6, 7])
@pytest.mark.parametrize("kind", ["random", "near_identity", "constant"])
@pytest.mark.parametrize("K", [70, 168, 252, 420])
def test_products_against_exact_sums(K, kind, S):
    """|O - exact| within the operands' rounding, the dropped levels (p pairs a level, digits of at most
    128), the last accumulator's rounding (S = 7) and the final one; the sums of levels 0 to 5 stay
    below 2^24, where FP32 accumulation is exact."""
    rng = np.random.default_rng(K)
    m = 4
    if kind == "random":
        A, B = (rng.standard_normal((m, K)) / np.sqrt(K) for _ in range(2))
        A /= np.linalg.norm(A, axis=1)[:, None]
        B /= np.linalg.norm(B, axis=1)[:, None]
    elif kind == "near_identity":
        A, B = (np.eye(m, K) * 0.999 + 1e-3 * rng.uniform(-1, 1, (m, K)) / np.sqrt(K) for _ in range(2))
    else:
        A, B = np.full((m, K), 1 / np.sqrt(K)), np.full((m, K), -0.93 / np.sqrt(K))
    dA, dB = (np.array([[digits(fixed(x, 0, S), S) for x in row] for row in M]) for M in (A, B))
    top = 7 if S == 7 else 5
    levels = [sum(dA[:, :, i] @ dB[:, :, l - i].T for i in range(max(0, l - S + 1), min(l, S - 1) + 1))
              for l in range(top + 1)]
    assert max(np.abs(l).max() for l in levels[:6]) < 1 << 24
    u = 2.0 ** -(bits_of(S) + 1)                               # operand rounding
    dropped = sum(2.0 ** (-8 * l) * (2 * S - 1 - l) * K for l in range(top + 1, 2 * S - 1))
    last = 2.0 ** -60 if S == 7 else 0.0                       # 2^24 2^-62 2^-24 and the cut to 2^-61
    for r in range(m):
        for c in range(m):
            got = join([int(l[r, c]) for l in levels], S)
            exact = sum(Fraction(a) * Fraction(b) for a, b in zip(A[r].tolist(), B[c].tolist()))
            norms = np.abs(A[r]).sum() + np.abs(B[c]).sum()
            bound = u * norms + K * u * u + dropped + last + 2.0 ** -61 + 2.0 ** -53 * abs(float(exact))
            assert abs(float(Fraction(got) - exact)) <= bound


def round_at(x, P):
    magic = {0: F32(12582912.0), 8: F32(49152.0), 16: F32(192.0), 24: F32(0.75)}[P]
    return (x + magic).astype(F32) - magic


def slice4f(h, l):
    q0 = round_at(h, 0)
    d = (h - q0).astype(F32)
    q1 = round_at((d + l).astype(F32), 8)
    d = ((d - q1).astype(F32) + l).astype(F32)
    q2 = round_at(d, 16)
    return [q0, q1, q2, round_at((d - q2).astype(F32), 24)]


def test_slices_of_unnormalised_pairs_are_bf16_and_restore_the_value():
    """h + l in units of 2^-8, |h| <= 256, |l| up to 2^-2: four BF16 numbers, their sum within half a
    unit of the last slice (2^-25) and the one rounded addition (2^-34 of them)."""
    rng = np.random.default_rng(1)
    h = np.concatenate([rng.uniform(-256, 256, 4000), [256, -256, 0, 255.99998, 0.5, -0.5]]).astype(F32)
    l = np.concatenate([rng.uniform(-0.25, 0.25, 4000), [0, 0, 0, 0.25, -0.25, 0.25]]).astype(F32)
    l[:2000] *= (2.0 ** rng.uniform(-24, 0, 2000)).astype(F32)
    q = slice4f(h, l)
    for j, x in enumerate(q):
        mant, _ = np.frexp(x.astype(np.float64))
        assert np.all(mant * 256 == np.rint(mant * 256)), j
    err = np.abs(sum(x.astype(np.float64) for x in q) - (h.astype(np.float64) + l.astype(np.float64)))
    assert err.max() <= 2.0 ** -25 + 2.0 ** -33


def test_level_join_is_exact_in_its_first_sum():
    """tc::join: a0 an integer, a1 a multiple of 2^-8 below 2^15, a2 ~2^3: s + e within the rounding of
    the terms at e's size, also where |a1| > |a0|."""
    rng = np.random.default_rng(2)
    a0 = np.rint(rng.uniform(-65536, 65536, 4000) * 2.0 ** rng.uniform(-16, 0, 4000)).astype(F32)
    a1 = (np.rint(rng.uniform(-32768, 32768, 4000) * 256 * 2.0 ** rng.uniform(-16, 0, 4000)) / 256).astype(F32)
    a2 = rng.uniform(-8, 8, 4000).astype(F32)
    assert np.any(np.abs(a1) > np.abs(a0))
    s = (a0 + a1).astype(F32)
    e0 = (a1 - (s - a0).astype(F32)).astype(F32)
    np.testing.assert_array_equal(s.astype(np.float64) + e0, a0.astype(np.float64) + a1)
    e = (e0 + a2).astype(F32)
    exact = a0.astype(np.float64) + a1 + a2
    assert np.abs(s.astype(np.float64) + e - exact).max() <= 2.0 ** -20  # half an ulp at 2^3 + 2^-8


def test_scaled_pairs_keep_the_product():
    """tc::scaled: coef (hi, lo) times v (hi, lo), not normalised: 2^-45 of the product."""
    rng = np.random.default_rng(3)
    c, v = rng.uniform(-1, 1, 4000) * 2.0 ** -8, rng.uniform(-65536, 65536, 4000)
    ch, vh = c.astype(F32), v.astype(F32)
    cl, vl = (c - ch).astype(F32), (v - vh).astype(F32)

    def fma(a, b, x):
        return (a.astype(np.float64) * b.astype(np.float64) + x.astype(np.float64)).astype(F32)

    p = (ch * vh).astype(F32)
    r = fma(cl, vh, fma(ch, vl, fma(ch, vh, -p)))
    exact = (ch.astype(np.float64) + cl) * (vh.astype(np.float64) + vl)
    assert np.all(np.abs(p.astype(np.float64) + r - exact) <= 2.0 ** -45 * np.abs(v) * 2.0 ** -8)
