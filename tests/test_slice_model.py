"""A NumPy model of the slice arithmetic of the tcgen05 GEMM (csrc/kernels_oz.cu),
step by step in float32, against exact integers and fractions: three slices (the
split precision) and six (FP64).

Three slices of a number relative to 2^E of its row, scaled to 2^15, in rounds of
1 to 4 octets of 8 complex (16 real terms each): the FP16 of a rest below 2^-5
(2^-17) and its FP32 rounding (2^-20), 2^-32 (1 + 1/8) of the row's scale; the sums
of (0, 0) and (0, 1) are exact in FP32.  Six digits of 9 bits: the FP16 of the sixth,
below 2^8, 2^-57 of the row's scale, and what is cut off before, 2^-60; class sums 0 to 3
and the carries between the classes are exact; sums over up to 512 rounds stay within
2^-57 of the largest partial sum."""
from fractions import Fraction

import numpy as np
import pytest

f32 = np.float32


def fma(a, b, c):  # products of two float32 are exact in float64; sums here need fewer than 53 bits
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(f32)


def half(x):
    return np.asarray(x, f32).astype(np.float16).astype(np.float64)


# ------------------------------------------------------------------ three slices
B = {1: 11, 2: 10, 3: 9, 4: 9}                      # bits of the second slice, by octets of the round
M1 = {1: f32(1.5 * 131072), 2: f32(1.5 * 262144), 3: f32(1.5 * 524288), 4: f32(1.5 * 524288)}


def slices3(x, E, octets):
    """oz_slice of float64 values x, |x| < 2^E: h + l with h = fl(x)."""
    h = x.astype(f32)
    l = (x - h).astype(f32)
    f, m0 = f32(2.0 ** (15 - E)), f32(1.5 * 2.0 ** 29)
    r = fma(h, f, m0)
    s0 = r - m0
    t = fma(l, f, fma(h, f, m0 - r))
    s1 = (t + M1[octets]) - M1[octets]
    return s0, s1, t - s1


@pytest.mark.parametrize("octets", [1, 2, 3, 4])
def test_three_slices(octets):
    rng = np.random.default_rng(octets)
    b = B[octets]
    x = np.concatenate([rng.uniform(-1, 1, 20000), rng.standard_normal(2000) * 2.0 ** rng.uniform(-40, 0, 2000) / 8,
                        1 - 2.0 ** -np.arange(1.0, 40), 2.0 ** -np.arange(1.0, 40), [0.0]])
    x = np.concatenate([x, -x])
    for E in (-90, 0, 7, 100):
        s0, s1, s2 = slices3(x * 2.0 ** E, E, octets)
        assert (np.abs(s0) <= 2.0 ** 15).all() and (s0 % 64 == 0).all()
        assert (np.abs(s1) <= 2.0 ** 5).all() and (s1 * 2.0 ** (b - 5) % 1 == 0).all()
        assert (np.abs(s2) <= 2.0 ** (4 - b)).all()
        assert np.array_equal(half(s0), s0) and np.array_equal(half(s1), s1)
        back = half(s0) + half(s1) + half(s2)
        # and x as two FP32 numbers, 2^-48
        assert np.abs(back * 2.0 ** -15 - x).max() <= 2.0 ** -32 + 2.0 ** -35 + 2.0 ** -48


@pytest.mark.parametrize("octets", [1, 2, 3, 4])
def test_three_slice_leading_sums_are_exact(octets):
    n, b = 16 * octets, B[octets]
    rng = np.random.default_rng(10 + octets)
    for k in range(40):
        if k == 0:      # the largest digits, and ones that leave the last bit odd
            a0, c0, a1 = np.full(n, 2.0 ** 15), np.full(n, 2.0 ** 15), np.full(n, 2.0 ** 5)
        else:
            a0, c0 = (64.0 * rng.integers(-512, 513, n) for _ in range(2))
            a1 = rng.integers(-2 ** b, 2 ** b + 1, n) * 2.0 ** (5 - b)
            a0[0], c0[0], a1[0] = 64.0, 64.0, 2.0 ** (5 - b)
            if k % 2:
                a0, c0, a1 = np.abs(a0), np.abs(c0), np.abs(a1)
        for u, v in ((a0, c0), (a0, a1)):
            s = f32(0)
            for p in u * v:
                s = f32(s + f32(p))
            assert float(s) == float(np.sum(u * v))


def test_three_slice_products():
    """|sum - exact| of one round over 64 real terms, classes i + j <= 3: 2 x 2^-32 x 9/8 of the row
    scales per term, s2 t2 (2^-40) and the FP32 sums of the rest (2^-41): below 64 x 2^-30.8."""
    rng = np.random.default_rng(3)
    for k in range(200):
        a, b = (rng.standard_normal(64) * 2.0 ** rng.uniform(-12 * (k % 3), 0, 64) for _ in range(2))
        ea, eb = (int(np.frexp(np.abs(x).max().astype(f32))[1]) for x in (a, b))
        sa, sb = ([half(s) for s in slices3(x, e, 4)] for x, e in ((a, ea), (b, eb)))
        got = sum(float(np.dot(sa[i], sb[j])) for i in range(3) for j in range(3) if i + j <= 3) * 2.0 ** -30
        exact = float(sum(Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b)) / Fraction(2) ** (ea + eb))
        assert abs(got - exact) < 64 * 2.0 ** -30.8


# ------------------------------------------------------------------ six slices
def digits6(x, E):
    """double_digits: five integers and the FP16 of the rest, value sum d_p 2^(-9p) 2^(E-8)."""
    F = int(Fraction(float(x)) * Fraction(2) ** (60 - E))  # towards zero
    d = []
    for p in range(5):
        k = 52 - 9 * p
        q = (F + (1 << (k - 1))) >> k
        F -= q << k
        d.append(q)
    return d, float(half(f32(F * 2.0 ** -7)))


def _samples(rng, n):
    x = np.concatenate([rng.uniform(-1, 1, n), rng.standard_normal(n) * 2.0 ** rng.uniform(-70, -3, n),
                        # digits of +-256 and +-255 one after the other
                        [512 / 513, -512 / 513, 256 / 513, 511 / 1022, 1 - 2.0 ** -53, 0.5, 2.0 ** -9, 0.0]])
    return np.concatenate([x, -x])


def test_six_digits():
    rng = np.random.default_rng(6)
    for E in (-1000, 0, 900):
        for x in _samples(rng, 400):
            y = np.ldexp(x, E)
            d, last = digits6(y, E)
            assert all(abs(q) <= 256 for q in d) and abs(last) <= 256
            back = sum(Fraction(q) / 512 ** p for p, q in enumerate(d)) + Fraction(last) / 512 ** 5
            assert abs(back / 256 - Fraction(float(y)) / Fraction(2) ** E) <= Fraction(9, 2 ** 60)
            for p in range(4):  # the remainder is at most half a unit, so an extreme digit turns the sign
                if abs(d[p]) == 256:
                    assert d[p] * d[p + 1] <= 0


def _class_sums(A, C):
    """Exact sums of the products of class 0 .. 6 (integers; the sixth digit in units of 2^-7)."""
    return [sum(int(A[p] @ C[c - p]) if p < 5 and c - p < 5 else float(A[p].astype(float) @ C[c - p].astype(float))
                for p in range(max(0, c - 5), min(c, 5) + 1)) for c in range(7)]


def _rows():
    """Digit rows [6][64] of two operands: the largest class sums there are."""
    rng = np.random.default_rng(8)
    alt = np.array([256, -256, 256, -256, 256, -256])[:, None] * np.ones((1, 64), int)
    top = 255 * np.ones((6, 64), int)
    one = np.array([255, 255, 255, 256, 0, 0])[:, None] * np.ones((1, 64), int)
    two = np.array([256, -255, -255, 256, 0, 255])[:, None] * np.ones((1, 64), int)
    kinds = [alt, -alt, top, -top, one, two, -two]
    for a in kinds:
        for c in kinds:
            yield a, c
            yield np.where(np.arange(64) < 32, a, alt), np.where(np.arange(64) < 32, c, alt)
    for _ in range(300):
        x = [_samples(rng, 64)[rng.integers(0, 272, 64)] for _ in range(2)]
        yield tuple(np.array([digits6(v, 0)[0] + [int(round(digits6(v, 0)[1]))] for v in y]).T for y in x)


def test_six_slice_class_sums_and_carries_are_exact():
    """Classes 0 to 3 are at most 2^24; class 3 with the carry of the classes above stays there too (an
    extreme product in class 3 makes two of class 4 oppose it), so tri_of's carries are exact."""
    W, MG, NM, NB = f32(2.0 ** -9), f32(1.5 * 2.0 ** 23), f32(-1.5 * 2.0 ** 23), f32(-512)

    def carry(x):
        return fma(x, W, MG) + NM

    for A, C in _rows():
        D = _class_sums(A, C)
        assert all(abs(D[c]) <= 2 ** 24 for c in range(4))
        for c in range(4):
            s = f32(0)
            for p in range(c + 1):
                for v in (A[p] * C[c - p]):
                    s = f32(s + f32(v))
            assert int(s) == D[c]
        d = [f32(x) for x in D]
        d4 = fma(fma(d[6], W, d[5]), W, d[4])
        c4 = carry(d4)
        assert abs(D[3] + int(c4)) <= 2 ** 24
        d3 = d[3] + c4
        c3 = carry(d3)
        d2 = d[2] + c3
        c2 = carry(d2)
        d1 = d[1] + c2
        c1 = carry(d1)
        a = d[0] + c1
        m = fma(fma(c1, NB, d1), f32(2.0 ** -9), fma(c2, NB, d2) * f32(2.0 ** -18))
        l = fma(fma(c3, NB, d3), f32(2.0 ** -27), fma(c4, NB, d4) * f32(2.0 ** -36))
        got = Fraction(float(a)) + Fraction(float(m)) + Fraction(float(l))
        exact = sum(Fraction(x) / 512 ** c for c, x in enumerate(D))
        # D4 to D6 are rounded to 24 bits: 2^-36 x (64 x 5 x 2^16) x 2^-24 and the last step's rounding
        assert abs(got - exact) <= Fraction(2) ** -34
        assert abs(float(m)) < 0.51 and abs(float(l)) < 0.51 * 2.0 ** -18


def _two_sum(a, b):
    s = f32(a + b)
    bb = f32(s - a)
    return s, f32(f32(a - f32(s - bb)) + f32(b - bb))


def test_sums_over_rounds():
    rng = np.random.default_rng(12)
    for R in (2, 8, 64, 512):
        for _ in range(50):
            h, m, l = f32(0), f32(0), f32(0)
            exact, top = Fraction(0), 0.0
            for _ in range(R):
                x = [f32(np.round(rng.uniform(-2.0 ** 22, 2.0 ** 22))), f32(rng.uniform(-0.5, 0.5)),
                     f32(rng.uniform(-0.5, 0.5) * 2.0 ** -18)]
                exact += sum(Fraction(float(v)) for v in x)
                h, e1 = _two_sum(h, x[0])
                mm, e2 = _two_sum(m, x[1])
                m, e3 = _two_sum(mm, e1)
                l = f32(f32(l + x[2]) + f32(e2 + e3))
                top = max(top, abs(float(h)), 2.0 ** 22)
            got = Fraction(float(h)) + Fraction(float(m)) + Fraction(float(l))
            assert abs(float(got - exact)) <= 2.0 ** -57 * top


def test_digits_of_a_normalised_sum():
    """tri_digits of h + m + l (each the rounded value of what is left).  What the two inner sums leave (2^-25) joins
    after three more digits as up to 2^-7: the fourth and the sixth digit may reach 256 + 4, and above 256 the FP16 of
    the sixth is 2^-56 of the row's scale; l joins the rest of the first sum, 2^-25, with 24 bits: 2^-58."""
    rng = np.random.default_rng(14)
    MG, Bf = f32(1.5 * 2.0 ** 23), f32(512)

    def digit(a, f):
        d = f32(MG - fma(a, f, MG))
        return d, fma(a, f, d)

    def fast(a, b):
        s = f32(a + b)
        return s, f32(b - f32(s - a))

    for x in _samples(rng, 3000):
        if abs(x) >= 1:
            continue
        h = f32(x)
        if abs(h) >= 1:
            continue
        m = f32(x - float(h))
        l = f32(rng.uniform(-0.5, 0.5) * 2.0 ** -24 * abs(float(m)))
        nf = f32(-256.0)
        s0, t = digit(h, nf)
        te = f32(m * nf)
        t, te = fast(t, te)
        te = fma(l, nf, te)
        s1, t = digit(t, Bf)
        s2, t = digit(t, Bf)
        te = f32(te * f32(262144))
        t, te = fast(t, te)
        s3, t = digit(t, Bf)
        s4, t = digit(t, Bf)
        s5 = fma(te, f32(-134217728), f32(t * f32(-512)))
        d = [s0, s1, s2, s3, s4]
        assert all(float(v) == round(float(v)) for v in d) and np.array_equal(half(d), d)
        assert all(abs(float(v)) <= 256 for v in (s0, s1, s2, s4)) and abs(float(s3)) <= 260 and abs(float(s5)) <= 260
        back = sum(Fraction(float(v)) / 512 ** p for p, v in enumerate(d)) + Fraction(float(half(s5))) / 512 ** 5
        exact = (Fraction(float(h)) + Fraction(float(m)) + Fraction(float(l))) * 256
        assert abs(back - exact) / 256 <= Fraction(5, 2 ** 58)
