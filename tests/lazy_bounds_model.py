"""Model of the lazy GF(M61) products in montmul_b200/csrc (mm_field.cuh, mm_kernels.cuh): the
squaring, the constant products, the weighted input and the wraparound half-pointwise step, as
maximum values. It checks that no intermediate passes 2^64, that each offset K p of a subtraction
covers the subtrahend, and that every value stored between passes is below 2^61 + 2^34.
tests/test_lazy_bounds.py runs it; test_wrapped_bounds.py checks the functions themselves and the
butterflies.
"""
P = (1 << 61) - 1
TOP = (1 << 64) - 1
class V:
    def __init__(s, m): assert 0 <= m <= TOP, hex(m); s.m = m
def add(a, b): return V(a.m + b.m)
def sub(a, b, K): assert K * P >= b.m, (K, hex(b.m)); return V(a.m + K * P)
def fold(x): return V(P + (x.m >> 61))
def mul1(a, b):  # (P & p) + (P >> 61), product < 2^125
    prod = a.m * b.m; assert prod < 1 << 125; return V(P + (prod >> 61))
class C:
    def __init__(s, re, im): s.re, s.im = re, im
def cadd(a, b): return C(add(a.re, b.re), add(a.im, b.im))
def cfold(x): return C(fold(x.re), fold(x.im))
W = V(P - 1)  # canonical constant
ONE = (1 << 61) + (1 << 34)
def inp(): return C(V(ONE), V(ONE))
def check_one(c, what):
    assert c.re.m <= ONE and c.im.m <= ONE, (what, hex(c.re.m), hex(c.im.m))

# ---- pointwise operations ----
def kmul_lazy_sums(x):
    """lkmulc: constants (wr, wi) canonical, s = wr + wi and d = wi - wr + p formed lazily."""
    s = add(W, W); d = sub(W, W, 1)
    k1 = mul1(add(x.re, x.im), W); k2 = mul1(x.re, d); k3 = mul1(x.im, s)
    return C(fold(sub(k1, k3, 4)), fold(add(k1, k2)))


def check_pointwise():
    # lsqr_scale with c = 4
    x = inp()
    re = fold(mul1(add(x.re, x.im), sub(x.re, x.im, 2)))
    t = mul1(x.re, x.im)
    im = fold(add(t, t))
    check_one(C(fold(V(re.m * 4)), fold(V(im.m * 4))), "square")
    # lreal_times: a 32-bit limb times a canonical constant
    check_one(C(fold(mul1(V((1 << 32) - 1), W)), fold(mul1(V((1 << 32) - 1), W))), "weighted input")
    check_one(kmul_lazy_sums(inp()), "kmul lazy sums")
    # half_pointwise: e = zp + conj zq, d = zp - conj zq, out = e A + d B
    zp, zq = inp(), inp()
    e = C(add(zp.re, zq.re), add(zp.im, sub(V(0), zq.im, 2)))
    d = C(sub(zp.re, zq.re, 2), add(zp.im, zq.im))
    check_one(cfold(cadd(kmul_lazy_sums(cfold(e)), kmul_lazy_sums(cfold(d)))), "half pointwise")
    # lkmul_re: re(x c) = x.re c.re + x.im (p - c.im)
    check_one(C(fold(add(mul1(V(ONE), W), mul1(V(ONE), W))), V(0)), "real only")
