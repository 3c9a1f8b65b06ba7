"""The link list of very large spheres (k_plinks, mglc_gb300/csrc/k_particle.cu), modelled:
its entries fit 31 bits (negative ones mean something else) and give node and direction
back, however many nodes a slab has and however the links lie."""
import math
import os
import random
import re

import pytest

SRC = open(os.path.join(os.path.dirname(__file__), "..", "mglc_gb300", "csrc", "k_particle.cu")).read()
PB, NSLAB, CAP = 256, 4, 256 * 27


def _span():
    m = re.search(r"constexpr int LINK_SPAN = 1 << (\d+);", SRC)
    return 1 << int(m.group(1)) if m else 1 << 62


def _walk(nbox, links_of_round, span):
    """The scan: yields (entry, node, direction) as entries are read back."""
    tb = nl = 0
    held = []
    for t0 in links_of_round.rounds(nbox):
        for t, a in links_of_round(t0):
            held.append(((t - tb) * 32 + a, t, a))
            nl += 1
        if nl <= CAP - PB * 18 and t0 + PB < nbox and t0 + 2 * PB - tb <= span:
            continue
        for entry, t, a in held:
            yield entry, t, a, tb
        held, nl, tb = [], 0, t0 + PB


class _Sparse:
    """Links in a few rounds only; rounds without any are walked at the list's limits."""

    def __init__(self, nbox, span, rng):
        n = (nbox + PB - 1) // PB
        near = [k for s in range(0, nbox, span) for k in range(s // PB - 2, s // PB + 3)]
        self.at = sorted({k for k in near + [0, 1, n - 2, n - 1] + [rng.randrange(n) for _ in range(40)]
                          if 0 <= k < n})
        self.nbox, self.rng = nbox, rng

    def rounds(self, nbox):
        return [k * PB for k in self.at]

    def __call__(self, t0):
        return [(t0 + i, a) for i in (0, PB - 1) for a in (1, 18) if t0 + i < self.nbox]


@pytest.mark.parametrize("radius", [5.0, 100.0, 319.0, 320.0, 330.5, 580.0])
def test_entries_fit_and_come_back(radius):
    bw = 2 * (math.ceil(radius) + 2) + 2
    nbox = bw * bw * max((s + 1) * bw // NSLAB - s * bw // NSLAB for s in range(NSLAB))
    assert nbox < 1 << 31
    seen = 0
    span = _span()
    for entry, t, a, tb in _walk(nbox, _Sparse(nbox, min(span, nbox), random.Random(3)), span):
        assert 0 <= entry < 1 << 31
        assert (tb + (entry >> 5), entry & 31) == (t, a)
        seen += 1
    assert seen > 8


def _s32(x):
    x &= (1 << 32) - 1
    return x - (1 << 32) if x >> 31 else x


def test_torque_sums_pass_32_bits():
    """Sphere of radius 250 centred at x = 2800: a thread's share of the top slab's
    sum m (n_z e_x - n_x e_z) stays in 32 bits, the slab's does not, and the kernel's sum
    from halves is exact."""
    rng = random.Random(7)
    R, cx, h = 250.0, 2800.0, 252
    threads = [0] * PB
    n = 0
    for z in range(125, h + 1):  # the links of every seventh column of the slab, weighed by 49
        for y in range(-h, h + 1, 7):
            for x in range(-h, h + 1, 7):
                if not R * R < x * x + y * y + z * z <= (R + 2) ** 2:
                    continue
                for m, e in ((2, (0, 0, -1)), (1, (1, 0, -1)), (1, (-1, 0, -1)), (1, (0, 1, -1)), (1, (0, -1, -1))):
                    if (x + e[0]) ** 2 + (y + e[1]) ** 2 + (z + e[2]) ** 2 <= R * R:
                        for _ in range(49):
                            threads[n % PB] += m * ((z + 300) * e[0] - int(x + cx) * e[2])
                            n += 1
    total = sum(threads)
    assert abs(total) >= 1 << 31 and max(abs(v) for v in threads) < 1 << 31
    got = 0
    for w in range(PB // 32):
        warp = threads[32 * w:32 * w + 32]
        lo = sum(v & 0xFFFF for v in warp)
        hi = sum(v >> 16 for v in warp)
        assert lo < 1 << 32 and abs(hi) < 1 << 31
        got += hi * 65536 + lo
    assert got == total
    assert re.search(r"const long long b = warp_sum64\(nt\[q\]\);", SRC)


@pytest.mark.gpu
def test_torque_does_not_depend_on_where_the_sphere_is():
    """The same sphere in a periodic channel near its start and near its end, where the
    slabs' sums pass 32 bits.  The sums' remainders are differences of numbers up to 2^32,
    a 18th of which rounds at 2^-53 in some four operations for each of four slabs, twice."""
    import numpy as np

    import mglc_gb300 as mg
    torque = []
    for x in (700.25, 7800.25):
        with mg.ParticleFlow(8000, 300, 300, [[x, 150.4, 150.7]], 140.0, tauf=0.65, rho_solid=1.2,
                             periodic_x=True, body_force=(1e-5, 0.0, 0.0), gravity=(0.0, 0.0, -1e-5),
                             threshold_wall=2.0, precision="fp32") as c:
            c.initial()
            c.step(1)
            torque.append(c.state()["torque"][0])
    assert np.abs(torque[0] - torque[1]).max() <= 4 * 4 * 2 * 2.0 ** (32 - 53) / 18
