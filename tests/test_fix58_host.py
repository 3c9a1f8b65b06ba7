"""The spheres' FP64 moments on integers (fix58_moments, mglc_gb300/csrc/k_particle.cu) and
in FP64 (mrt_moments, lbm_common.cuh), both modelled with exact rationals: the same bits
for every cell that the integer form takes.  The FP64 statements name their fused
multiply-adds where a product is not exact, so the bits are not the compiler's choice."""
import os
import random
import re
from fractions import Fraction as Fr

CSRC = os.path.join(os.path.dirname(__file__), "..", "mglc_gb300", "csrc")
ONE = 1 << 58


def rn(x):
    return Fr(float(x))  # Fraction to float rounds to nearest even


def rn53(v):
    hi = v >> 32
    r = max(11 - (32 - (hi ^ (hi >> 63)).bit_length()), 0)
    m = (1 << r) - 1
    return (v + (m >> 1) + ((v >> r) & m & 1)) & ~m


class F64:
    """FP64: every operation rounds once."""

    def __init__(self, x):
        self.x = Fr(x)

    def __add__(self, o):
        return F64(rn(self.x + o.x))

    def __sub__(self, o):
        return F64(rn(self.x - o.x))

    @staticmethod
    def fma(c, a, b):
        return F64(rn(c * a.x + b.x))

    @staticmethod
    def mul(c, a):
        return F64(rn(c * a.x))

    def value(self):
        return self.x


class I58:
    """Units of 2^-58, each sum rounded to 53 bits."""

    def __init__(self, v):
        self.v = v

    def __add__(self, o):
        return I58(rn53(self.v + o.v))

    def __sub__(self, o):
        return I58(rn53(self.v - o.v))

    @staticmethod
    def fma(c, a, b):
        assert abs(c * a.v + b.v) < 1 << 63
        return I58(rn53(c * a.v + b.v))

    @staticmethod
    def mul(c, a):
        assert abs(c * a.v) < 1 << 63
        return I58(rn53(c * a.v))

    def value(self):
        return Fr(self.v, ONE)


def moments(f):
    T = type(f[0])
    pairs = [(1, 2), (3, 4), (5, 6), (7, 10), (9, 8), (11, 14), (13, 12), (15, 18), (17, 16)]
    s = [None] + [f[a] + f[b] for a, b in pairs]
    d = [None] + [f[a] - f[b] for a, b in pairs]
    sa, se = s[1] + s[2] + s[3], (s[4] + s[5]) + (s[6] + s[7]) + (s[8] + s[9])
    a45, b45, a67, b67, a89, b89 = d[4] + d[5], d[4] - d[5], d[6] + d[7], d[6] - d[7], d[8] + d[9], d[8] - d[9]
    sxy, sxz, syz = s[4] + s[5], s[6] + s[7], s[8] + s[9]
    s23, t23, sp, sm = s[2] + s[3], s[2] - s[3], sxy + sxz, sxy - sxz
    return [T.fma(-30, f[0], T.fma(8, se, T.mul(-11, sa))), T.fma(12, f[0], T.fma(-4, sa, se)),
            T.fma(-4, d[1], a45 + a67), T.fma(-4, d[2], b45 + a89), T.fma(-4, d[3], b67 + b89),
            T.fma(-2, syz, T.fma(2, s[1], T.mul(-1, s23)) + sp),
            T.fma(-2, syz, T.fma(-4, s[1], T.mul(2, s23)) + sp), t23 + sm, T.fma(-2, t23, sm),
            s[4] - s[5], s[8] - s[9], s[6] - s[7], a45 - a67, a89 - b45, b67 - b89]


def test_integer_moments_are_the_fp64_ones():
    rng = random.Random(9)
    w = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
    for k in range(400):
        spread = rng.choice([1e-6, 0.02, 0.3])
        f = [x * (1 + rng.uniform(-spread, spread)) for x in w]
        if k % 4 == 0:  # the corners of the range
            f = [rng.choice([2.0 ** -6, 0.12499999999999999, rng.uniform(2.0 ** -6, 0.125)]) for _ in w]
            f[0] = rng.choice([2.0 ** -6, 0.49999999999999994, rng.uniform(2.0 ** -6, 0.5)])
        assert all(Fr(x) * ONE == int(Fr(x) * ONE) for x in f)
        a = moments([F64(x) for x in f])
        b = moments([I58(int(Fr(x) * ONE)) for x in f])
        assert [x.value() for x in a] == [x.value() for x in b]


def test_fp64_statements_name_their_roundings():
    src = open(os.path.join(CSRC, "lbm_common.cuh")).read()
    body = src[src.index("MrtMom<T> mrt_moments("):src.index("void mrt_relax(")]
    coefs = set(re.findall(r"(?:T\((-?\d+)\)|\b(two|four))\s*\*", body))
    assert coefs <= {("-4", ""), ("", "two"), ("", "four")}  # powers of two only
    assert "__fma_rn(-30.0, f0, __fma_rn(8.0, se, __dmul_rn(-11.0, sa)))" in src
    assert "__fma_rn(12.0, f0, __fma_rn(-4.0, sa, se))" in src
    k = open(os.path.join(CSRC, "k_particle.cu")).read()
    assert "rn53(-30 * F[0].v + rn53(8 * se.v + rn53(-11 * sa.v)))" in k
    assert "rn53(12 * F[0].v + rn53(-4 * sa.v + se.v))" in k
