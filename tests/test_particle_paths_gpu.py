"""Branches of the sphere step against the general path.

FP64 cells take the integer form of the forward transform while f_1..18 lie in
[2^-6, 2^-3) and f_0 in [2^-6, 1/2), the FP64 form otherwise: rho0 = 0.5625 puts the
diagonal weights on the lower limit, 1.5 the rest weight and 2.25 the axis weights
on the upper ones (cells of both kinds side by side), 8 takes every cell to the FP64
form.  The bounds are those of the unit-density flow: 1e-10 on the populations,
1e-9 on the particle state."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_util import rel_l2
from tests.test_particle_gpu import CASE, mg  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

CENTERS = [[8.3, 11.7, 10.1], [21.6, 11.4, 10.2], [34.2, 10.8, 9.5]]


def _flow(mg, precision, centers=CENTERS, **over):
    kw = dict(CASE, nx=37, ny=23, nz=21)
    kw.update(over)
    nx, ny, nz, r = kw.pop("nx"), kw.pop("ny"), kw.pop("nz"), kw.pop("radius")
    kw["periodic_x"] = bool(kw["periodic_x"])
    return mg.ParticleFlow(nx, ny, nz, centers, r, precision=precision, **kw)


@pytest.mark.parametrize("rho0", [0.5625, 1.5, 2.25, 8.0])
def test_density_ranges_match_oracle(mg, rho0):  # noqa: F811
    over = dict(nx=37, ny=23, nz=21, rho0=rho0, rho_solid=1.2 * rho0)
    o = O.ParticleOracle(np.array(CENTERS), dim=3, qmode=1, **dict(CASE, **over))
    assert o.step(30) == 0
    ref = o.get()
    with _flow(mg, "fp64", **over) as c:
        c.initial()
        c.step(30)
        st, mask, f = c.state(), c.mask(), c.get_f()
    fluid = ref["obst"] == 0
    assert np.array_equal(mask < 0, fluid)
    assert rel_l2(f[fluid], ref["f"][fluid]) <= 1e-10
    for a, b in (("uc", "uc"), ("omega", "om"), ("force", "force"), ("torque", "torque")):
        assert rel_l2(st[a], ref[b]) <= 1e-8, a


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("g", [-0.05, -0.06])
def test_frozen_state_is_the_failing_steps(mg, precision, g):  # noqa: F811
    """A sphere that falls into the wall freezes the same state whether the steps
    come one by one or as many more in one call than were needed, an even or an
    odd number (the mask buffers alternate)."""
    over = dict(gravity=(0.0, 0.0, g), spring_scale_wall=0.0)
    centers = [[8.3, 11.7, 5.3], [21.6, 11.4, 10.2]]

    def run(chunks):
        with _flow(mg, precision, centers, **over) as c:
            c.initial()
            n = 0
            with pytest.raises(mg.MglcError):
                for k in chunks:
                    c.step(k)
                    n += k
            return n, c.mask(), c.state()

    n, mask, st = run([1] * 200)
    assert 0 < n < 199
    for extra in (n + 6, n + 7):
        _, m2, s2 = run([extra])
        assert np.array_equal(mask, m2)
        for k in ("xc", "uc", "omega"):
            assert np.array_equal(st[k], s2[k]), k


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp32", 1e-4)])
@pytest.mark.parametrize("rho0", [1.0, 2.0])
def test_node_refilled_in_the_first_step(mg, rho0, precision, tol):  # noqa: F811
    """A node just inside the sphere leaves it in the first step; its refill takes the
    average density of the collided populations, which start from w whatever rho0 is."""
    over = dict(nx=37, ny=23, nz=21, rho0=rho0, rho_solid=1.2 * rho0, gravity=(0.0, 0.0, 0.05))
    centers = [[18.0, 12.0, 10.499]]  # node (18, 12, 7) is 3.499 away
    o = O.ParticleOracle(np.array(centers), dim=3, qmode=1, **dict(CASE, **over))
    inside = o.get()["obst"][6, 11, 17]
    assert o.step(1) == 0
    ref = o.get()
    assert inside != 0 and ref["obst"][6, 11, 17] == 0
    with _flow(mg, precision, centers, **over) as c:
        c.initial()
        c.step(1)
        f = c.get_f()[6, 11, 17]
    assert np.abs(f - ref["f"][6, 11, 17]).max() <= tol * rho0


def _contacts(case):
    """80 spheres of radius 1.5 out of each other's reach but for four (with spaces of 33
    and 72 between their numbers) around sphere 5.  Offsets are multiples of 1/16:
    differences and squares are exact."""
    offsets = {0: ([3.0, 1.0, 0.5], [-3.0, 1.25, 0.5], [0.5, -3.0, 1.0], [0.75, 1.0, 3.125]),
               1: ([2.0, 2.0, 1.5], [-2.0, 2.0, -1.5], [1.5, -2.0, 2.0], [-1.75, -2.5, -0.75])}[case]
    at = [[4.0 + 4.25 * i, 4.0 + 4.25 * j, 4.0 + 4.25 * k] for k in range(4) for j in range(4) for i in range(5)]
    focus = np.array([36.0, 12.0, 12.0])
    at[5] = list(focus)
    for c2, o in zip((0, 33, 72, 41), offsets):
        at[c2] = list(focus + o)
    return np.array(at), focus


@pytest.mark.parametrize("case", [0, 1])
def test_contact_forces_are_added_in_a_stated_order(mg, case):  # noqa: F811
    """Lane l of 32 adds the springs of particles l, l + 32, ..., then the lanes' sums by
    halves: bit for bit, whatever number of threads looks for contacts."""
    at, focus = _contacts(case)
    r, thr = 1.5, 1.0
    over = dict(nx=48, ny=24, nz=24, radius=r, threshold_particle=thr, threshold_wall=0.5,
                gravity=(0.0, 0.0, 0.0), body_force=(0.0, 0.0, 0.0))
    total = {}
    for scale in (0.0, 0.7):
        with _flow(mg, "fp64", at, spring_scale_particle=scale, **over) as c:
            c.initial()
            c.step(1)
            total[scale] = c.state()["force"][5]
    lanes = np.zeros((32, 3))
    for c2 in range(len(at)):
        d = focus - at[c2]
        dij = np.sqrt((d * d).sum())
        if c2 != 5 and dij < 2 * r + thr:
            t = (dij - r - r - thr) / thr
            lanes[c2 % 32] += 0.7 * (t * t) * d / dij
    assert np.count_nonzero(lanes.any(1)) == 4
    half = 16
    while half:
        lanes[:half] = lanes[:half] + lanes[half:2 * half]
        half //= 2
    assert np.array_equal(total[0.7], total[0.0] + lanes[0])
