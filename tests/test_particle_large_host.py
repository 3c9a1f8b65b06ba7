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
