"""Interval model of the lazy GF(M61^2) butterflies in montmul_b200/csrc/mm_ntt.cuh (ldif8, ldit8,
ldif4, ldit4, ldif2, ldit2): sums and differences without offsets are u64 values modulo 2^64 whose
true value lies in an interval, K p is added where the value is folded or rotated next. Checks, with
the kernels' exact sequences, offsets and fold points, that every interval is narrower than 2^64,
that whatever is folded or rotated is in [0, 2^64), and that everything stored is below
2^61 + 2^34. The products around them are lazy_bounds_model.py's. CPU only."""
import pytest

P = (1 << 61) - 1
ONE = (1 << 61) + (1 << 34)


class I:
    """A u64 modulo 2^64 whose true value lies in [lo, hi]."""

    def __init__(self, lo, hi):
        assert hi - lo < 1 << 64, (hex(lo), hex(hi))
        self.lo, self.hi = lo, hi

    def __add__(self, o):
        return I(self.lo + o.lo, self.hi + o.hi)

    def __sub__(self, o):
        return I(self.lo - o.hi, self.hi - o.lo)

    def plus(self, k):
        return I(self.lo + k * P, self.hi + k * P)

    def whole(self):
        assert self.lo >= 0 and self.hi < 1 << 64, (hex(self.lo), hex(self.hi))
        return self


def fold(x):
    return I(0, P + (x.whole().hi >> 61))


def rot(x):
    return I(0, P + (x.whole().hi >> 31))


class C:
    def __init__(self, re, im):
        self.re, self.im = re, im


def add(a, b, k=0):
    return C((a.re + b.re).plus(k), (a.im + b.im).plus(k))


def sub(a, b, k=0):
    return C((a.re - b.re).plus(k), (a.im - b.im).plus(k))


def sub_i(a, b):
    return C(b.im - a.im, a.re - b.re)


def add_mi(u, v, k=0):
    return C((u.re + v.im).plus(k), (u.im - v.re).plus(k))


def sub_mi(u, v, k=0):
    return C((u.re - v.im).plus(k), (u.im + v.re).plus(k))


def cfold(x):
    return C(fold(x.re), fold(x.im))


def w8(x):
    return C(rot((x.re - x.im).plus(3)), rot((x.re + x.im).plus(3)))


def inp(top=ONE):
    return C(I(0, top), I(0, top))


def stored(c):
    f = cfold(c)
    assert f.re.hi <= ONE and f.im.hi <= ONE


def dif8(x):
    a0, b0 = add(x[0], x[4]), sub(x[0], x[4])
    a1, b1 = cfold(add(x[1], x[5])), w8(sub(x[1], x[5]))
    a2, b2 = add(x[2], x[6]), sub_i(x[2], x[6])
    a3, b3 = cfold(add(x[3], x[7])), w8(sub_i(x[3], x[7]))
    c0, c2, c1, c3 = add(a0, a2), sub(a0, a2), add(a1, a3), sub_i(a1, a3)
    d0, d2, d1, d3 = add(b0, b2), sub(b0, b2), add(b1, b3), sub_i(b1, b3)
    return [add(c0, c1), sub(c0, c1, 3), add(c2, c3, 4), sub(c2, c3, 4),
            add(d0, d1, 3), sub(d0, d1, 5), add(d2, d3, 4), sub(d2, d3, 4)]


def dit8(x):
    c0, c1, c2, c3 = add(x[0], x[1]), sub(x[0], x[1]), add(x[2], x[3]), sub(x[2], x[3])
    c4, c5, c6, c7 = add(x[4], x[5]), cfold(sub(x[4], x[5], 2)), add(x[6], x[7]), sub(x[6], x[7])
    a0, a2, a1, a3 = add(c0, c2), sub(c0, c2), add_mi(c1, c3), sub_mi(c1, c3)
    b0, b2 = cfold(add(c4, c6)), cfold(sub(c4, c6, 3))
    b1, b3 = add_mi(c5, c7), sub_mi(c5, c7)
    v1 = C(rot((b1.re + b1.im).plus(3)), rot((b1.im - b1.re).plus(4)))
    v3 = C(rot((b3.im - b3.re).plus(4)), rot((I(0, 0) - b3.re - b3.im).plus(5)))
    return [add(a0, b0), add(a1, v1, 3), add_mi(a2, b2, 4), add(a3, v3, 3),
            sub(a0, b0, 2), sub(a1, v1, 4), sub_mi(a2, b2, 4), sub(a3, v3, 4)]


def dif4(x):
    a0, b0, a1, b1 = add(x[0], x[2]), sub(x[0], x[2]), add(x[1], x[3]), sub_i(x[1], x[3])
    return [add(a0, a1), sub(a0, a1, 3), add(b0, b1, 3), sub(b0, b1, 3)]


def dit4(x):
    c0, c1, c2, c3 = add(x[0], x[1]), sub(x[0], x[1]), add(x[2], x[3]), sub(x[2], x[3])
    return [add(c0, c2), add_mi(c1, c3, 3), sub(c0, c2, 3), sub_mi(c1, c3, 3)]


def dif2(x):
    return [add(x[0], x[1]), sub(x[0], x[1], 2)]


@pytest.mark.parametrize("f, r", [(dif8, 8), (dit8, 8), (dif4, 4), (dit4, 4), (dif2, 2)])
def test_butterfly_intervals(f, r):
    for y in f([inp() for _ in range(r)]):
        stored(y)


def test_model_rejects_what_would_wrap():
    """Unfolded sums of eight inputs are a hair too wide, and a short offset leaves a negative."""
    with pytest.raises(AssertionError):
        I(0, 4 * ONE) - I(0, 4 * ONE)
    with pytest.raises(AssertionError):
        stored(sub(inp(), inp(), 1))
