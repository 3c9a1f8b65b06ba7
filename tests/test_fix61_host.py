"""The integer arithmetic of the FP64 collision (mglc_gb300/csrc/fix61.cuh),
modelled with Python integers and compared with exact rational arithmetic:
loading is exact over the range that the kernel takes, storing rounds to
nearest even, a product by a coefficient is within 0.5 + 2^-20 units of
2^-61, and one lid collision lies closer to the exact one than the same
collision evaluated in FP64 (rms over random states and relaxation times).
Bounds: a population is the sum of two products (0.5 units each and the
roundings of its equilibrium, at most 6 units together), then half an ulp of
the result: at most 12 units + ulp/2."""
import math
import random
import struct
from fractions import Fraction as Fr

import pytest

import test_pair_form_host as P

ONE = 1 << 61
M32 = (1 << 32) - 1


def s32(x):
    x &= M32
    return x - (1 << 32) if x >> 31 else x


def load(x):
    b = struct.unpack("<Q", struct.pack("<d", x))[0]
    hi, lo = b >> 32, b & M32
    s = (hi >> 20) - 1014
    mh = (hi & 0xFFFFF) | 0x100000
    return ((((mh << 32) | lo) << s) >> 32 & M32) << 32 | (lo << s) & M32


def store(v):
    hi = v >> 32
    lz = 32 - hi.bit_length()
    r = 11 - lz
    w = v + ((1 << (r - 1)) - 1) + ((v >> r) & 1)
    return struct.unpack("<d", struct.pack("<Q", (w >> r) + ((1024 - lz) << 52)))[0]


def coef(c):
    C = round(Fr(c) * (1 << 64))
    assert abs(C) < 1 << 63
    low = s32(C)
    return (C - low) >> 32, low


def mad(v, c, a):
    h, low = c
    vl = s32(v)
    vh = (v >> 32) + ((vl & M32) >> 31)
    x = vh * low + (0x80000000 + (vl * low >> 32)) + vl * h
    assert abs(x) < 1 << 63
    return vh * h + a + (x >> 32)


def in_range(rng):
    return rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-8, -2)


def test_load_is_exact_and_store_rounds_to_nearest_even():
    rng = random.Random(1)
    xs = [2.0 ** -8, math.nextafter(0.5, 0), 0.25, math.nextafter(0.25, 0), 1 / 36, 1 / 18, 1 / 3]
    for x in xs + [in_range(rng) for _ in range(2000)]:
        assert Fr(load(x)) == Fr(x) * ONE
        assert store(load(x)) == x
    for k in range(20000):
        L = rng.randint(54, 63)
        v = rng.getrandbits(L - 1) | 1 << (L - 1)
        if k % 3 == 0:  # ties and their neighbours
            r = L - 53
            v = (v >> r << r) + (1 << (r - 1)) + rng.choice([-1, 0, 1])
        assert store(v) == float(Fr(v, ONE)), v


@pytest.mark.parametrize("c", [0.4999, -0.4999, 1 / 3, 1e-9, -0.25, 0.0])
def test_product_is_rounded_to_nearest(c):
    rng = random.Random(2)
    h, low = coef(c)
    assert abs(Fr(h * (1 << 32) + low, 1 << 64) - Fr(c)) <= Fr(1, 1 << 65)
    for k in range(4000):
        v = rng.choice([1, -1]) * rng.getrandbits(rng.randint(1, 61))
        a = rng.randint(-(1 << 60), 1 << 60)
        err = Fr(mad(v, (h, low), a) - a) - Fr(v) * Fr(h * (1 << 32) + low, 1 << 64)
        assert abs(err) <= Fr(1, 2) + Fr(1, 1 << 20)


def mul(v, w, S):
    (vh, vl), (wh, wl) = v, w
    x = vh * wl + ((1 << (S - 33)) + (vl * wl >> 32)) + vl * wh
    assert abs(x) < 1 << 63 and abs(vh * wh << (64 - S)) < 1 << 63
    return (vh * wh << (64 - S)) + (x >> (S - 32))


def dig(v):
    assert abs(v) < 1 << 63
    vl = s32(v)
    return (v - vl) >> 32, vl


def recip(rho, seed_error=0.0):
    x = round(float(1 / Fr(rho, ONE)) * (1 + seed_error) * 2 ** 28)
    h, low = dig(rho)
    e = ONE - ((h * x << 4) + (low * x >> 28))
    assert abs(e >> 10) < 1 << 31
    x1 = (x << 32) + (x * (e >> 10) >> 19)
    e1 = ONE - mul(dig(rho), dig(x1), 60)
    assert abs(e1) < 1 << 31
    return x1 + ((x1 >> 32) * e1 + (1 << 28) >> 29)


def test_reciprocal():
    rng = random.Random(4)
    for k in range(4000):
        rho = rng.randint(ONE // 4, ONE * 11 // 4)
        got = recip(rho, rng.uniform(-1, 1) * 2.0 ** -22)
        assert abs(Fr(got) - Fr(1 << 121, rho)) <= Fr(3, 2)


PAIRS = P.PAIRS


def fixed_lid(f, snu, sq):
    """fix61_collide_lid on the loaded populations."""
    F = [load(x) for x in f]
    e = P.E.astype(int)
    r, j = sum(F), [sum(int(e[q][a]) * F[q] for q in range(19)) for a in range(3)]
    snu, sq = Fr(snu), Fr(sq)
    c1, c2, l18, l6 = coef((1 - snu) / 2), coef((1 - sq) / 2), coef(snu / 36), coef(sq / 12)
    inv = recip(r, 2.0 ** -24)
    u = [dig(mul(dig(a), dig(inv), 58)) for a in j]
    k = [dig(mad(a, coef(snu / 4), 0)) for a in j]
    X, Y, Z = (mul(k[a], u[a], 64) for a in range(3))
    cxy, cxz, cyz = 2 * mul(k[0], u[1], 64), 2 * mul(k[0], u[2], 64), 2 * mul(k[1], u[2], 64)
    qh = mul(dig(mad(Y - Z, coef(Fr(1, 6)), 0)), dig((1 << 60) - inv), 60)
    S = X + Y + Z
    b = mad(r, l18, mad(S, coef(Fr(-1, 3)), 0))
    gx, gy, gz = (mad(a, l6, 0) for a in j)
    bxy, bxz, byz = b + qh + X + Y, b - qh + X + Z, b + Y + Z
    E = [2 * b + 2 * X, 2 * b - 2 * qh + 2 * Y, 2 * b + 2 * qh + 2 * Z, bxy + cxy, bxy - cxy,
         bxz + cxz, bxz - cxz, byz + cyz, byz - cyz]
    O = [2 * gx, 2 * gy, 2 * gz, gx + gy, gx - gy, gx + gz, gx - gz, gy + gz, gy - gz]
    out = [0] * 19
    out[0] = 2 * mad(F[0], c1, mad(r, coef(snu / 6), -2 * S))
    for (p, q), ev, od in zip(PAIRS, E, O):
        s, t = mad(F[p] + F[q], c1, ev), mad(F[p] - F[q], c2, od)
        out[p], out[q] = s + t, s - t
    return out


def exact_lid(f, snu, sq):
    """The pair form (equal to the moment form: test_pair_form_host) in rationals."""
    f = [Fr(x) for x in f]
    e = P.E.astype(int)
    snu, sq = Fr(snu), Fr(sq)
    rho, j = sum(f), [sum(int(e[q][a]) * f[q] for q in range(19)) for a in range(3)]
    u = [a / rho for a in j]
    usq = sum(a * a for a in u)
    q6 = (u[1] ** 2 - u[2] ** 2) * (rho - 1) / 12
    w = [Fr(1, 3)] + [Fr(1, 18)] * 6 + [Fr(1, 36)] * 12
    out = [f[0] - snu * (f[0] - w[0] * (rho - Fr(3, 2) * rho * usq))] + [Fr(0)] * 18
    for n, (p, q) in enumerate(PAIRS):
        eu = sum(int(e[p][a]) * u[a] for a in range(3))
        E = 2 * w[p] * rho * (1 + Fr(9, 2) * eu * eu - Fr(3, 2) * usq)
        E += [0, -q6, q6, q6 / 2, q6 / 2, -q6 / 2, -q6 / 2, 0, 0][n]
        O = 6 * w[p] * rho * eu
        ne, no = f[p] + f[q] - E, f[p] - f[q] - O
        out[p], out[q] = f[p] - snu / 2 * ne - sq / 2 * no, f[q] - snu / 2 * ne + sq / 2 * no
    return out


def test_collision_is_closer_to_exact_than_fp64():
    rng = random.Random(3)
    sums = [0.0, 0.0]
    for _ in range(300):
        tau = 0.5 + 10 ** rng.uniform(-3, 0.3)
        snu, sq = 1.0 / tau, 8 * (2 * tau - 1) / (8 * tau - 1)
        u = [rng.uniform(-0.15, 0.15) for _ in range(3)]
        rho = 1.0 + rng.uniform(-0.03, 0.03)
        f = []
        for q in range(19):
            eu = sum(P.E[q][a] * u[a] for a in range(3))
            f.append(float(rho * P.W[q] * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * sum(a * a for a in u)) *
                           (1 + rng.uniform(-0.05, 0.05))))
        if not all(2.0 ** -8 <= x < (0.5 if q == 0 else 0.125) for q, x in enumerate(f)):
            continue
        want, got = exact_lid(f, snu, sq), fixed_lid(f, snu, sq)
        r = sum(f)
        ref = P.pair_lid(P.np.array(f), r, r, P.np.array([sum(P.E[q][a] * f[q] for q in range(19))
                                                          for a in range(3)]) / r, snu, sq)
        for q in range(19):
            v = store(got[q]) if got[q] >= 1 << 53 else float(Fr(got[q], ONE))
            err = abs(Fr(v) - want[q])
            assert err <= Fr(12, ONE) + Fr(math.ulp(v)) / 2
            sums[0] += float(err) ** 2
            sums[1] += float(abs(Fr(float(ref[q])) - want[q])) ** 2
    assert sums[0] < sums[1], (math.sqrt(sums[0]), math.sqrt(sums[1]))


def test_sums_round_like_fp64():
    """rn53 (macro64.cuh) after an exact integer sum is FP64's rounding of that sum."""
    def rn53(v):
        hi = v >> 32
        r = max(11 - (32 - (hi ^ (hi >> 63)).bit_length()), 0)
        m = (1 << r) - 1
        return (v + (m >> 1) + ((v >> r) & m & 1)) & ~m

    rng = random.Random(6)
    for k in range(20000):
        v = rng.choice([1, -1]) * rng.getrandbits(rng.randint(1, 62))
        if k % 3 == 0 and abs(v) > 1 << 55:  # ties
            r = abs(v).bit_length() - 53
            v = (v >> r << r) + (1 << (r - 1))
        elif k % 5 == 0:
            v = rng.choice([1, -1]) << rng.randint(50, 62)
        assert Fr(rn53(v), ONE) == Fr(float(Fr(v, ONE))), v
