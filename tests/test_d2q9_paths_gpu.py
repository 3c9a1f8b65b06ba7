"""The D2Q9 collision's fast path and the statements it stands for
(mglc_gb300/csrc/d2q9.cuh): bitwise against the oracle on states that sit on
either side of its range checks, on rows that do not fill a warp."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mg():
    from mglc_gb300 import build
    build.build()
    import mglc_gb300
    return mglc_gb300


def _state(kind, ny, nx, rng):
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    f = w * (1.0 + 1e-2 * (rng.random((ny, nx, 9)) - 0.5))
    if kind == "rest":  # zero momenta, zero relaxed moments
        f = np.broadcast_to(w, (ny, nx, 9)).copy()
    elif kind == "tiny":  # below 2^-900: no two-term reciprocal
        f *= 2.0 ** -950
    elif kind == "huge":
        f *= 2.0 ** 940
    elif kind == "zeros":  # zero and negative-zero populations
        f[:, ::2, 1:] = 0.0
        f[::3, 1::2, 5:] = -0.0
    elif kind == "ones":  # densities whose significand is all ones
        f[:] = 0.0
        f[..., 0] = np.where(rng.random((ny, nx)) < 0.5, 1.0 - 2.0 ** -53, 2.0 - 2.0 ** -52)
    elif kind == "specials":
        f[1, 1, 3] = np.inf
        f[ny - 1, nx - 1, 5] = np.nan
    return f


@pytest.mark.parametrize("kind", ["flow", "rest", "tiny", "huge", "zeros", "ones", "specials"])
@pytest.mark.parametrize("nx,ny", [(2, 3), (33, 7), (129, 5)])
def test_lid2d_matches_oracle_bitwise(mg, kind, nx, ny):
    f = _state(kind, ny, nx, np.random.default_rng(nx + len(kind)))
    o = O.Lid2DOracle(nx, ny, 200.0, 0.1)
    with mg.LidDrivenCavity2D(nx, ny, reynolds=200.0, u0=0.1) as c, np.errstate(all="ignore"):
        c.load_state(f)
        rho, u, v = c.macro()
        o.f[:], o.rho[:], o.u[:], o.v[:] = f, rho, u, v
        for _ in range(3):
            c.step(1)
            o.run(1)
            got, want = c.get_f(), o.f
            assert np.array_equal(got, want, equal_nan=True)
            fin = ~np.isnan(want)
            assert np.array_equal(np.signbit(got[fin]), np.signbit(want[fin]))


def test_frozen_state_keeps_its_mask(mg):
    """A circle that runs into a wall: the failing step leaves the mask it started with,
    and so does every later call."""
    with mg.ParticleFlow2D(40, 40, [[20.0, 7.5]], 6.0, gravity=0.5) as c:
        c.initial()
        with pytest.raises(mg.MglcError):
            c.step(200)
        m, xc = c.mask(), c.state()["xc"][0]
        j, i = np.mgrid[1:41, 1:41]
        assert np.array_equal(m >= 0, (i - xc[0]) ** 2 + (j - xc[1]) ** 2 <= 36.0)
        for n in (1, 2, 3):
            with pytest.raises(mg.MglcError):
                c.step(n)
            assert np.array_equal(c.mask(), m)
        c.initial()
        c.step(1)
        assert (c.mask() >= 0).sum() > 0


@pytest.mark.parametrize("kind", ["diagonal", "rest", "axis", "thin", "dense"])
def test_lid2d_integer_sums_bitwise(mg, kind):
    """Populations on either side of the range in which the sums run on integers
    ([2^-6, 1/4), the rest population up to 1/2, density from 1/4): the limits
    themselves, their neighbours and mixed cells."""
    rng = np.random.default_rng(11)
    nx, ny = 67, 5
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    f = w * (1.0 + 0.2 * (rng.random((ny, nx, 9)) - 0.5))

    def around(limit, n):  # the limit, its neighbours and values close by
        near = np.array([limit, np.nextafter(limit, 0), np.nextafter(limit, 1)])
        pick = rng.integers(0, 4, (ny, nx, n))
        return np.where(pick < 3, near[np.minimum(pick, 2)], limit * (1 + 0.1 * (rng.random((ny, nx, n)) - 0.5)))

    if kind == "diagonal":
        f[..., 5:] = around(2.0 ** -6, 4)
    elif kind == "rest":
        f[..., :1] = around(0.5, 1)
    elif kind == "axis":
        f[..., 1:5] = around(0.25, 4)
    elif kind == "thin":  # densities around 1/4 from populations in range
        f = np.array([0.08] + [0.021] * 8) * (1.0 + 0.1 * (rng.random((ny, nx, 9)) - 0.5))
    else:  # the largest density in range
        f[..., 0] = np.nextafter(0.5, 0)
        f[..., 1:] = np.where(rng.random((ny, nx, 8)) < 0.8, np.nextafter(0.25, 0), 0.2)
    o = O.Lid2DOracle(nx, ny, 200.0, 0.1)
    with mg.LidDrivenCavity2D(nx, ny, reynolds=200.0, u0=0.1) as c:
        c.load_state(f)
        rho, u, v = c.macro()
        o.f[:], o.rho[:], o.u[:], o.v[:] = f, rho, u, v
        for _ in range(3):
            c.step(1)
            o.run(1)
            assert np.array_equal(c.get_f(), o.f)
