"""The lazy GF(M61^2) arithmetic of the kernels stays within 64 bits: the functions themselves (the
butterflies of montmul_b200/csrc/mm_ntt.cuh, the products of mm_field.cuh, the half-length pointwise step of
mm_kernels.cuh), built for the host with g++ over intervals in place of uint64_t. A value is a u64 modulo
2^64 whose true value lies in an interval narrower than 2^64; whatever is folded, rotated or multiplied
has to lie in [0, 2^64), and whatever is stored between passes below 2^61 + 2^34. The outputs of each
butterfly go through the product that follows it, and product outputs into the next butterfly. Only the
bit operations (lfold, lrot, lmul1) are modelled by their bounds. CPU only."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "montmul_b200", "csrc")

MODEL = r'''
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#define __device__
#define __forceinline__ inline
typedef __int128 i128;
static const char* where = "";
static void need(bool ok, const char* what) {
    if (!ok) { std::printf("%s: %s\n", where, what); std::exit(1); }
}
struct V {
    i128 lo, hi;
    V(long long c = 0) : lo(c), hi(c) {}
    V(i128 l, i128 h) : lo(l), hi(h) { need(h - l < (i128)1 << 64, "wider than 2^64"); }
    const V& whole() const { need(lo >= 0 && hi < (i128)1 << 64, "not in [0, 2^64)"); return *this; }
};
static V operator+(V a, V b) { return V(a.lo + b.lo, a.hi + b.hi); }
static V operator-(V a, V b) { return V(a.lo - b.hi, a.hi - b.lo); }
static V operator*(V a, V b) {   // of constants, and of a value in [0, 2^64) by a small factor
    need((a.lo == a.hi || b.lo == b.hi) && a.whole().hi < (i128)1 << 62 && b.whole().hi < (i128)1 << 62, "product");
    return V(a.lo * b.lo, a.hi * b.hi);
}
static const i128 P = ((i128)1 << 61) - 1, ONE = ((i128)1 << 61) + ((i128)1 << 34);
static const V P2((long long)P);
static V lfold(V x) { return V(0, P + (x.whole().hi >> 61)); }
static V lrot(V x) { return V(0, P + (x.whole().hi >> 31)); }
static V lmul1(V a, V b) {
    const unsigned __int128 p = (unsigned __int128)a.whole().hi * (unsigned __int128)b.whole().hi;
    need(p >> 125 == 0, "product of 125 bits");
    return V(0, P + (i128)(p >> 61));
}
struct F2 { V re, im; };
struct F2K { V re, im, s, d; };
static F2 f2(V re, V im) { return F2{re, im}; }
static int swz(int e) { return e; }
static void half_pair(int, int& p, int& q) { p = 0; q = 1; }
#define uint64_t V
@FUNCTIONS@
#undef uint64_t
static const V C(0, P - 1);   // a canonical constant
static const F2K W{C, C, C, C};
static F2 in() { return F2{V(0, ONE), V(0, ONE)}; }
static F2 stored(F2 x) {
    need(x.re.whole().hi <= ONE && x.im.whole().hi <= ONE, "stored above 2^61 + 2^34");
    return x;
}
template <int R> static void passes(const char* dif, const char* dit) {
    for (int tw = 0; tw < 2; ++tw) {
        F2 x[R];
        for (auto& v : x) v = in();
        where = dif;
        ldif<R>(x);
        for (int k = 0; k < R; ++k) stored(tw && k ? lkmul(stored(lcfold(x[k])), W) : lcfold(x[k]));
        where = dit;
        for (int k = 0; k < R; ++k) x[k] = tw && k ? stored(lkmul(in(), W)) : in();
        ldit<R>(x);
        for (auto& v : x) stored(v);
    }
}
int main() {
    passes<8>("dif8", "dit8");
    passes<4>("dif4", "dit4");
    passes<2>("dif2", "dit2");
    where = "square";
    for (uint32_t c = 1; c <= 4; ++c) stored(lsqr_scale(in(), c));
    where = "products";
    stored(lkmulc(in(), F2{C, C}));
    stored(F2{lkmul_re(in(), W), V(0)});
    where = "half-length pointwise";
    F2 z[2] = {in(), in()}, ab[4] = {{C, C}, {C, C}, {C, C}, {C, C}};
    half_pointwise_pair(z, 2, ab, 0);
    stored(z[0]);
    stored(z[1]);
    std::printf("ok\n");
}
'''


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def function(text, pattern):
    """One function of a source: from the start of the line that matches to its closing brace."""
    m = re.search(r"^[^\n]*" + pattern, text, re.M)
    assert m, pattern
    end = depth = text.index("{", m.end())
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
            return text[m.start():end] + "\n"


def functions():
    field, ntt, kern = source("mm_field.cuh"), source("mm_ntt.cuh"), source("mm_kernels.cuh")
    out = [function(field, rf"\b{n}\(") for n in ("lsub", "lcfold", "lcadd", "lkmul", "lkmulc", "lkmul_re", "lsqr_scale")]
    start = ntt.index("template <int K> __device__ __forceinline__ uint64_t lsum(")
    end = ntt.index("template <int R> __device__ __forceinline__ void ldif(F2* x)")
    out.append(ntt[start:end])
    out += [function(ntt, rf"void {n}\(F2\* x\)") for n in ("ldif", "ldit")]
    out.append(function(kern, r"void half_pointwise_pair\(F2\* s2, int H"))
    return "".join(out)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("bounds")

    def run(text):
        (d / "b.cpp").write_text(MODEL.replace("@FUNCTIONS@", text))
        subprocess.run([gxx, "-std=c++17", "-w", str(d / "b.cpp"), "-o", str(d / "b")], check=True)
        return subprocess.run([str(d / "b")], capture_output=True, text=True).stdout.strip()

    return run


def test_lazy_arithmetic_stays_in_64_bits(check):
    assert check(functions()) == "ok"


# An offset one short, a fold left out: each would wrap in the kernels.
@pytest.mark.parametrize("old,new,where", [
    ("a1 = lcfold(wadd(x[1], x[5]))", "a1 = wadd(x[1], x[5])", "dif8"),
    ("x[5] = wsub_k<5>(d0, d1)", "x[5] = wsub_k<4>(d0, d1)", "dif8"),
    ("lrot(5 * P2 - b3.re - b3.im)", "lrot(4 * P2 - b3.re - b3.im)", "dit8"),
    ("c5 = lcfold(wsub_k<2>(x[4], x[5]))", "c5 = lcfold(wsub_k<1>(x[4], x[5]))", "dit8"),
    ("x[3] = wsub_k<3>(b0, b1)", "x[3] = wsub_k<2>(b0, b1)", "dif4"),
    ("x[1] = lcfold(wsub_k<2>(u, x[1]))", "x[1] = lcfold(wsub_k<1>(u, x[1]))", "dit2"),
    ("lfold(lsub<3>(k1, k3))", "lfold(lsub<1>(k1, k3))", "dif8"),
    ("zp.im + lsub<2>(0, zq.im)", "zp.im + lsub<1>(0, zq.im)", "half-length pointwise"),
])
def test_a_change_that_would_wrap_is_seen(check, old, new, where):
    text = functions()
    assert text.count(old) >= 1
    assert check(text.replace(old, new, 1)).startswith(where + ":")
