"""The arithmetic of the sliced contractions (csrc/fire_sliced.cu) and of the determinant Laplacian's FP32 sums (DlSum in
csrc/fire_det.cu), restated in numpy and Python integers and checked against exact sums, with error bounds from the formats.

SL_PAIR: a row (column) is scaled by 2^(6 - e), e the exponent of its largest magnitude, to x in (-128, 128), and cut into six
slices, x = s_0 + s_1 2^-9 + ..., s_0 = rint(x), |s_i| <= 256; the last one keeps FP16's 11 bits (2^-49 of x at most, 2^-55 of
the largest magnitude, which is 64 at least).  Levels l = i + j < 6 are summed exactly; the ones left out are at most
5 2^16 2^-54 per product (level 6, five pairs of 2^8 2^8) and a 2^-9 th of that per level beyond.
SL_F64: eight balanced base-256 digits of x 2^56 rounded to an integer; levels l < 8; what is left out is at most
7 2^14 2^-64 per product and less beyond; one rounding to 53 bits at the end.
Both bounds are relative to the product of the largest magnitudes, not to the terms."""
from fractions import Fraction

import numpy as np
import pytest

from test_compensated_sum import grid_sum

f32, f64, LD = np.float32, np.float64, np.longdouble
ZERO, NAN = -32768, 32767


# ------------------------------------------------------------------------------------------------ SL_PAIR
def _codes32(m):
    f = (m.astype(f32).view(np.int32) >> 23) & 0xff
    return np.where(m == 0, ZERO, np.where(f == 255, NAN, np.maximum(f - 127, -119)))


def _slices32(A, axis):
    bits = np.abs(A).view(np.uint32).max(axis)  # of the bit patterns: a NaN is the largest
    code = _codes32(bits.view(f32))
    c = np.expand_dims(code, axis)
    inv = np.where((c == ZERO) | (c == NAN), 0.0, np.ldexp(1.0, np.where(abs(c) > 300, 0, 6 - c))).astype(f32)
    x = np.where(np.isfinite(A), A, 0) * inv
    out = []
    for i in range(6):
        s = np.rint(x) if i < 5 else x.astype(np.float16).astype(f32)
        assert np.all(np.abs(s) <= (128 if i == 0 else 256)) and np.all(s == s.astype(np.float16))
        out.append(s.astype(f64))
        x = ((x - s) * f32(512)).astype(f32)
    return out, code


def _scale(code):
    return np.where(code == ZERO, 0.0, np.where(code == NAN, np.nan, np.ldexp(1.0, np.where(abs(code) > 300, 0, code - 6))))


def _two_sum(a, b):
    s = (a + b).astype(f32)
    v = (s - a).astype(f32)
    return s, ((a - (s - v).astype(f32)).astype(f32) + (b - v).astype(f32)).astype(f32)


def pair(A, B):
    """hi + lo of A @ B, as the tensor core and the epilogue form them."""
    sa, ra = _slices32(A, 1)
    sb, cb = _slices32(B, 0)
    hi = lo = None
    for k in range(0, A.shape[1], 256):
        L = [sum(sa[i][:, k:k + 256] @ sb[l - i][k:k + 256] for i in range(l + 1)) for l in range(6)]
        assert all(np.all(np.abs(L[l]) <= 1 << 24) for l in (0, 1))  # exact in FP32
        L = [x.astype(f32) for x in L]
        low = (L[3] + ((L[4] + (L[5] * f32(2.0**-9))).astype(f32) * f32(2.0**-9))).astype(f32) * f32(2.0**-27)
        h, e = _two_sum(L[0], L[1] * f32(2.0**-9))
        h, e2 = _two_sum(h, L[2] * f32(2.0**-18))
        l = ((e + e2).astype(f32) + low).astype(f32)
        if hi is None:
            hi, lo = h, l
        else:
            hi, e = _two_sum(hi, h)
            lo = (lo + (e + l).astype(f32)).astype(f32)
    sc = _scale(ra)[:, None] * _scale(cb)[None]
    return hi.astype(f64) * sc, lo.astype(f64) * sc


# ------------------------------------------------------------------------------------------------ SL_F64
def _digits(A, axis):
    """Base-256 digits (highest first) of every value on its row's (column's) grid, and the exponents."""
    m = np.abs(A).max(axis)
    code = np.where(m > 0, np.frexp(m)[1] - 1, ZERO).astype(int)
    c = np.broadcast_to(np.expand_dims(code, axis), A.shape)
    out = np.zeros((8,) + A.shape)
    for ix in np.ndindex(A.shape):
        if c[ix] == ZERO:
            continue
        v = Fraction(float(A[ix])) * Fraction(2) ** int(62 - c[ix])
        q0 = q = (abs(v.numerator) * 2 // v.denominator + 1) // 2 * (1 if v >= 0 else -1)  # halves away from zero
        assert abs(q) < 1 << 63
        for i in range(7, 0, -1):
            d = (q + 128) % 256 - 128
            out[i][ix] = d
            q = (q - d) >> 8
        out[0][ix] = q
        assert abs(q) <= 128 and sum(int(out[i][ix]) << (8 * (7 - i)) for i in range(8)) == q0
    return out, code


def assemble(value, e):
    """sl_assemble: value = h 2^32 + l (96 bits), times 2^e, as a double."""
    h, l = value >> 32, value & 0xffffffff
    neg = h < 0
    if neg:
        h, l = ~h, l ^ 0xffffffff  # one's complement
    x, y, z, up = h >> 32, h & 0xffffffff, l, 0
    if x == 0:
        x, y, z, up = y, z, 0, 32
    if x == 0:
        x, y, up = y, 0, 64
    if x == 0:
        return 0.0
    lz = 32 - x.bit_length()
    m = (((x << 64 | y << 32 | z) << lz) >> 32) & ((1 << 64) - 1)
    ex = e + 32 - up - lz  # value = m 2^ex, bit 63 of m set
    field = ex + 1086
    drop = 11 if field > 0 else 12 - field
    q = 0 if drop > 64 else (m >> drop) + ((m >> (drop - 1)) & 1)
    bits = 0x7ff << 52 if field > 2046 else ((field - 1) << 52) + q if field > 0 else q
    r = float(np.array(bits, np.uint64).view(f64))
    return -r if neg else r


def f64_sliced(A, B):
    da, ra = _digits(A, 1)
    db, cb = _digits(B, 0)
    out = np.zeros((A.shape[0], B.shape[1]))
    total = np.zeros(out.shape, object)
    for l in range(8):
        L = sum(da[i] @ db[l - i] for i in range(l + 1))
        if l <= 3 and A.shape[1] <= 256:
            assert np.all(np.abs(L) <= 1 << 24)
        total = total + np.vectorize(int, otypes=[object])(L) * 256 ** (7 - l)
    for ix in np.ndindex(out.shape):
        if ra[ix[0]] != ZERO and cb[ix[1]] != ZERO:
            out[ix] = assemble(total[ix], int(ra[ix[0]] + cb[ix[1]] - 68))
    return out


def _operands(name, rng):
    K = 512 if name == "two chunks" else 256
    A, B = rng.normal(size=(12, K)), rng.normal(size=(K, 9)) / 16
    if name == "activations":
        A = A / (1 + np.exp(-A))
    elif name == "cancelling":
        B[K // 2:] = -B[:K // 2] * (1 + 1e-3 * rng.normal(size=(K // 2, 9)))
        A[:, K // 2:] = A[:, :K // 2]
    elif name == "scaled":
        A *= 10.0 ** rng.uniform(-25, 8, (12, 1))
        B *= 10.0 ** rng.uniform(-8, 8, (1, 9))
    return A.astype(f32), B.astype(f32)


CASES = ["normal", "activations", "cancelling", "scaled", "two chunks"]


@pytest.mark.parametrize("name", CASES)
def test_pair_sums(name):
    A, B = _operands(name, np.random.default_rng(3))
    exact = A.astype(LD) @ B.astype(LD)
    top = np.abs(A).max(1)[:, None].astype(f64) * np.abs(B).max(0)[None]
    hi, lo = pair(A, B)
    err = np.abs(hi.astype(LD) + lo - exact).astype(f64)
    K = A.shape[1]
    # per product, in units of x x' (2^12 at least where both are the largest): levels left out, the last slices' ends; then
    # the pair's own rounding, 2^-47 of the level sums (at most the result's magnitude plus 2^-8 of K top)
    per = (5 * 2.0**-38 * 1.01 + 2 * 2.0**-49 * 128) / 2.0**12
    assert np.all(err <= K * per * top + 2.0**-47 * (np.abs(exact).astype(f64) + K * top / 256))
    # no further off than the sums of the CUDA cores
    comp = grid_sum(A, B)
    comp = comp[0] if isinstance(comp, tuple) else comp
    assert (err / top).max() <= (np.abs(np.asarray(comp).astype(LD) - exact).astype(f64) / top).max()


@pytest.mark.parametrize("name", CASES)
def test_f64_sums(name):
    A, B = (x[:6, :] if i == 0 else x[:, :5] for i, x in enumerate(_operands(name, np.random.default_rng(4))))
    rng = np.random.default_rng(5)
    A, B = A.astype(f64) * (1 + 1e-9 * rng.normal(size=A.shape)), B.astype(f64) * (1 + 1e-9 * rng.normal(size=B.shape))
    top = np.abs(A).max(1)[:, None] * np.abs(B).max(0)[None]
    got = f64_sliced(A, B)
    plain = A @ B
    K = A.shape[1]
    per = (7 * 2.0**-50 * 1.01 + 2 * 2.0**-57 * 128) / 2.0**12
    worst = 0.0
    for ix in np.ndindex(got.shape):
        exact = sum(Fraction(float(a)) * Fraction(float(b)) for a, b in zip(A[ix[0]], B[:, ix[1]]))
        err = float(abs(Fraction(float(got[ix])) - exact))
        assert err <= K * per * top[ix] + 2.0**-53 * abs(float(exact)) * 1.001
        worst = max(worst, err / top[ix])
    ref = max(float(abs(Fraction(float(plain[ix])) - sum(Fraction(float(a)) * Fraction(float(b))
                                                         for a, b in zip(A[ix[0]], B[:, ix[1]])))) / top[ix]
              for ix in np.ndindex(got.shape))
    assert worst <= ref  # of the plain FP64 sums


def test_what_the_bound_is_relative_to():
    """Large values of a row against zero weights, the sum carried by values 2^-30 below: within the bound, which is relative to
    the largest magnitudes, but far from the value's own rounding.  Rows like that (envelope coefficients) take other sums, whose
    grid follows every 16 k."""
    rng = np.random.default_rng(9)
    A = rng.uniform(0.5, 1.0, (8, 64)).astype(f32)
    A[:, 32:] *= f32(2.0**-30)
    B = rng.normal(size=(64, 5)).astype(f32)
    B[:32] = 0
    exact = (A.astype(LD) @ B.astype(LD)).astype(f64)
    hi, lo = pair(A, B)
    err = np.abs(hi + lo - exact)
    top = np.abs(A).max(1)[:, None] * np.abs(B).max(0)[None].astype(f64)
    assert np.all(err <= 64 * 2.0**-49 * top)
    assert np.any(err > 2.0**-24 * np.abs(exact))
    comp = grid_sum(A, B)
    comp = comp[0] if isinstance(comp, tuple) else comp
    assert np.all(np.abs(np.asarray(comp).astype(f64) - exact) <= 2.0**-40 * (np.abs(A).astype(f64) @ np.abs(B)))


def test_assembly_rounds_once():
    """Every length of the 96-bit sum, both signs, carries into the next power of two, and results that are denormal, zero or
    beyond the largest double."""
    rng = np.random.default_rng(6)
    values = [0, 1, -1, (1 << 53) - 1, (1 << 54) - 1, -((1 << 54) - 1), (1 << 94) - 1, -(1 << 94)]
    values += [int(rng.integers(1, 1 << 62)) * (-1) ** k >> int(rng.integers(0, 62)) for k in range(200)]
    values += [(int(rng.integers(1 << 30, 1 << 31)) << 62 | int(rng.integers(0, 1 << 62))) * (-1) ** k >> int(rng.integers(0, 90))
               for k in range(400)]
    for v in values:
        for e in (-68, 0, -1100, 1000):
            exact = Fraction(v) * Fraction(2) ** e
            got = assemble(v, e)
            if np.isinf(got):
                assert abs(exact) >= Fraction(2) ** 1024 * (1 - Fraction(1, 1 << 53))
                continue
            # half a unit in the last place (2^-1075 where that is denormal), and one unit of the sum (one's complement)
            tol = max(abs(exact) / (1 << 53), Fraction(1, 1 << 1075)) + Fraction(2) ** e
            assert abs(Fraction(got) - exact) <= tol, (v, e)


def test_rows_of_zeros_infinities_and_nans():
    rng = np.random.default_rng(7)
    A, B = rng.normal(size=(6, 32)).astype(f32), rng.normal(size=(32, 5)).astype(f32)
    clean = pair(A, B)
    A[1], B[:, 2] = 0, 0
    A[2, 5], A[3, 7], B[9, 4] = np.inf, np.nan, -np.inf
    hi, lo = pair(A, B)
    bad = np.zeros((6, 5), bool)
    bad[2], bad[3], bad[:, 4] = True, True, True
    assert np.all(np.isnan(hi[bad]))
    zero = np.zeros((6, 5), bool)
    zero[1], zero[:, 2] = True, True
    assert np.all(hi[zero & ~bad] == 0)
    keep = ~bad & ~zero
    assert np.array_equal(hi[keep], clean[0][keep]) and np.array_equal(lo[keep], clean[1][keep])


# ------------------------------------------------------------------------------------------------ DlSum<float>
def _fma(a, b, c):
    return f32(f64(a) * f64(b) + f64(c))  # the low part of a product: exact in double


def dl_sum(a, b):
    """The three-term expansion; non-finite where a product or a sum overflowed (the kernel then sums in double)."""
    s0 = s1 = s2 = f32(0)
    with np.errstate(all="ignore"):
        for x, y in zip(a, b):
            p = f32(x * y)
            h, hl = _two_sum(np.asarray(s0), np.asarray(p))
            l, ll = _two_sum(np.asarray(s1), np.asarray(_fma(x, y, -p)))
            m, ml = _two_sum(l, hl)
            s0, s1, s2 = f32(h), f32(m), f32(s2 + f32(ll + ml))
        return f64(s0) + (f64(s1) + f64(s2))


@pytest.mark.parametrize("scale", [1.0, 1e-10, 1e-16, 1e-20, 1e15])
def test_expansion_of_fp32_products(scale):
    """No less than a double keeps: 2^-53 of the largest partial sum, whatever is lost of the products' low parts below
    2^-149 each (products below 2^-102)."""
    rng = np.random.default_rng(8)
    for n in (1, 7, 64, 600):
        a = (scale * rng.normal(size=n) * 10.0 ** rng.uniform(-4, 4, n)).astype(f32)
        b = (scale * rng.normal(size=n)).astype(f32)
        if n > 7:
            a[n // 2:n // 2 * 2], b[n // 2:n // 2 * 2] = a[:n // 2], -b[:n // 2]
        prods = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b)]
        top, s = Fraction(0), Fraction(0)
        for q in prods:
            s += q
            top = max(top, abs(s), abs(q))
        assert abs(Fraction(float(dl_sum(a, b))) - s) <= top / (1 << 53) + n * Fraction(1, 1 << 149)


def test_expansion_says_when_it_overflowed():
    a, b = np.array([1e20, 1.0], f32), np.array([3e19, 2.0], f32)
    assert not np.isfinite(dl_sum(a, b))
    assert not np.isfinite(dl_sum(np.array([np.nan, 1], f32), b)) and not np.isfinite(dl_sum(np.array([np.inf, 1], f32), b))
    assert np.isfinite(dl_sum(np.array([1e18, -1e18], f32), np.array([1e19, 1e19], f32)))
