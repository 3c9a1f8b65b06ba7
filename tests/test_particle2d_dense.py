"""Circles of one node three apart: eight nodes of nine are fluid with a solid
neighbour, so the list of boundary nodes and their link terms is as long as it gets."""
import os
import re

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_particle2d_gpu import mg  # noqa: F401  (fixture)

SRC = os.path.join(os.path.dirname(__file__), "..", "mglc_gb300", "csrc", "k_particle2d.cu")
KW = dict(tauf=0.7, rho_solid=1.05, threshold_wall=0.2, threshold_particle=0.5)


def _centers(n):
    at = np.arange(2, n, 3.0)
    c = np.array([[x, y] for y in at for x in at])
    return c + np.random.default_rng(1).uniform(-0.03, 0.03, c.shape)


def _oracle(n, qmode=1):
    c = _centers(n)
    return O.ParticleOracle(np.c_[c, np.zeros(len(c))], dim=2, nx=n, ny=n, nz=1, radius=0.6,
                            gravity=(0.0, -1e-4, 0.0), qmode=qmode, **KW)


@pytest.mark.parametrize("n", [9, 60])
def test_link_terms_hold_every_listed_node(n):
    """The last term of the last listed node lies inside the array as it is allocated."""
    obst = np.pad(_oracle(n).get()["obst"][0], 1)
    near = sum(np.roll(obst, s, (0, 1)) for s in ((a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)))
    listed = int(((obst == 0) & (near > 0))[1:-1, 1:-1].sum())
    assert listed == n * n * 8 // 9
    src = open(SRC).read()
    names = dict(NODE_LINKS=8, LINK_TERMS=3, NODE_TERMS=24)
    size = eval(re.search(r"dal\(c, &d\.lt, ([^,]+), err\)", src).group(1), dict(names, nodes=n * n))
    assert 24 * (listed - 1) + 23 < size


@pytest.mark.gpu
@pytest.mark.parametrize("qmode", [0, 1])
@pytest.mark.parametrize("n", [9, 60])
def test_dense_circles_match_oracle_bitwise(mg, n, qmode):  # noqa: F811
    o = _oracle(n, qmode)
    assert o.step(6) == 0
    r = o.get()
    with mg.ParticleFlow2D(n, n, _centers(n), 0.6, gravity=1e-4, q_bisection=qmode == 0, **KW) as c:
        c.initial()
        c.step(6)
        f, (rho, u, v), st, m = c.get_f(), c.macro(), c.state(), c.mask()
    assert np.array_equal(f, r["f"][0])
    assert np.array_equal(rho, r["rho"][0]) and np.array_equal(u, r["u"][0]) and np.array_equal(v, r["v"][0])
    assert np.array_equal((m >= 0).astype(np.int32), r["obst"][0])
    for a, b in (("xc", "xc"), ("uc", "uc"), ("omega", "om"), ("force", "force"), ("torque", "torque")):
        assert np.array_equal(st[a], r[b]), a
