"""Temperatures of any scale in the FP64 heated cavity (mglc_gb300/csrc/fix61.cuh,
fix_heat): a cell's temperature populations are integers in units that its largest one
sets.  Modelled with Python integers, one collision is closer to the exact one (rms)
than its evaluation in FP64, from temperatures of 1e-300 to 1e3 and over the
diffusivities that the lattice takes; on the GPU, walls of 1e-9 to 300 against the
oracle, bounded relative to the temperature (the oracle's own rounding:
test_fix61_gpu.py, 30 * 30 * 2^-53 of the largest value a step)."""
import math
import random
import struct
from fractions import Fraction as Fr

import numpy as np
import pytest

import test_fix61_host as H
from oracle import oracle as O
from tests.test_fix61_gpu import _macros, _state, mg  # noqa: F401  (fixture)

QD, QNU = 3.0 - math.sqrt(3.0), 4.0 * math.sqrt(3.0) - 6.0


def _bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def _load(x, top):
    b = _bits(x)
    e = (b >> 52) & 0x7FF
    m = ((b & ((1 << 52) - 1)) | 1 << 52) << 10
    v = ((m >> min(top + 2 - e, 63)) + 1) >> 1
    return -v if b >> 63 else v


def _store(v, top):
    if v == 0:
        return 0.0
    b = _bits(float(v))
    assert 1 <= ((b >> 52) & 0x7FF) + top - 1082 < 2047
    return struct.unpack("<d", struct.pack("<Q", b + ((top - 1082) << 52)))[0]


def _weights(kappa):
    a = 42.0 * math.sqrt(3.0) * kappa - 6.0
    return a, [(1.0 - a) / 7.0] + [(a + 6.0) / 42.0] * 6


def _fixed(g, u, a):
    most = max(abs(1.0 - a) / 7.0, abs(6.0 + a) / 42.0)
    head = 0 if most >= 0.6 else 1 if most >= 0.3 else 2
    top = max((_bits(abs(x)) >> 52) for x in g) + head
    G = [_load(x, top) for x in g]
    T = sum(G)
    assert abs(T) < H.ONE
    g1, g2 = H.coef((1 - Fr(QNU)) / 2), H.coef((1 - Fr(QD)) / 2)
    c0, gE, hd = H.coef(Fr(QNU * (1.0 - a) / 7.0) / 4), H.coef(Fr(0.5 * QNU * (6.0 + a) / 21.0)), H.coef(Fr(QD) / 4)
    E, h = H.mad(T, gE, 0), H.dig(2 * H.mad(T, hd, 0))
    out = [2 * H.mad(G[0], g1, 2 * H.mad(T, c0, 0))] + [0] * 6
    for k in range(3):
        q = 2 * k + 1
        p = H.mad(G[q] + G[q + 1], g1, E)
        m = H.mad(G[q] - G[q + 1], g2, H.mul(h, H.dig(round(Fr(u[k]) * (1 << 63))), 63))
        out[q], out[q + 1] = p + m, p - m
    return [_store(v, top) for v in out]


def _pair(g, u, a, num):
    """pair_collide_t in the arithmetic num converts to."""
    qd, qnu, aa = num(QD), num(QNU), num(a)
    T = sum(num(x) for x in g)
    ge0, gE, gd = num(QNU * (1.0 - a) / 7.0), num(0.5 * QNU * (6.0 + a) / 21.0), qd / 2
    E, h = T * gE, T * gd
    out = [(1 - qnu) * num(g[0]) + T * ge0] + [num(0)] * 6
    for k in range(3):
        q = 2 * k + 1
        p = (num(1) / 2 - qnu / 2) * (num(g[q]) + num(g[q + 1])) + E
        m = (num(1) / 2 - qd / 2) * (num(g[q]) - num(g[q + 1])) + h * num(u[k])
        out[q], out[q + 1] = p + m, p - m
    return out


@pytest.mark.parametrize("kappa", [1e-3, 0.01, 0.035, 0.05, 0.08, 0.095])
def test_collision_is_closer_to_exact_than_fp64_at_any_scale(kappa):
    rng = random.Random(11)
    a, w = _weights(kappa)
    for scale in (1e-300, 1e-9, 1e-3, 0.3, 0.5, 1.0, 300.0, 1e3):
        sums = [0.0, 0.0]
        for _ in range(150):
            T = scale * rng.uniform(0.1, 1.0) * rng.choice([1, -1])
            g = [T * x * (1 + rng.uniform(-0.05, 0.05)) for x in w]
            u = [rng.uniform(-0.15, 0.15) for _ in range(3)]
            want, got, fp = _pair(g, u, a, Fr), _fixed(g, u, a), _pair(g, u, a, float)
            sums[0] += sum(float((Fr(x) - y) / Fr(scale)) ** 2 for x, y in zip(got, want))
            sums[1] += sum(float((Fr(x) - y) / Fr(scale)) ** 2 for x, y in zip(fp, want))
        assert sums[0] < sums[1], (scale, math.sqrt(sums[0]), math.sqrt(sums[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("ekman", [0.0, 1e-3])
@pytest.mark.parametrize("walls", [(1e-3, -1e-3), (1e-9, -1e-9), (1.0, 0.0), (300.0, 280.0)])
def test_walls_of_any_scale_match_oracle(mg, walls, ekman, in_place):  # noqa: F811
    nx, ny, nz = 35, 5, 6
    rng = np.random.default_rng(21)
    f = _state("flow", (nz, ny, nx), 8)
    lo, hi = min(walls), max(walls)
    T = lo + (hi - lo) * rng.random((nz, ny, nx))
    g = T[..., None] * (np.array([0.64] + [0.06] * 6)) * (1 + 0.02 * (rng.random((nz, ny, nx, 7)) - 0.5))
    m, T = _macros(f), g.sum(-1)
    t_ref = 0.5 * (lo + hi)
    o = O.ThermalOracle(nx, ny, nz, 1e5, 0.71, 0.1, ekman, *walls, t_ref)
    o.f[:], o.g[:], o.T[:], o.rho[:] = f, g, T, m[0]
    o.u[:], o.v[:], o.w[:] = m[1:]
    with mg.BuoyancyCavity(nx, ny, nz, rayleigh=1e5, prandtl=0.71, mach=0.1, t_hot=walls[0],
                           t_cold=walls[1], t_ref=t_ref, ekman=ekman, in_place=in_place) as c:
        c.load_state(f, g)
        for n in (1, 2, 3, 4):
            c.step(1)
            o.run(1)
            for got, want in zip(c.get_f(), (o.f, o.g)):
                assert np.abs(got - want).max() <= n * 900 * 2.0 ** -53 * np.abs(want).max()
