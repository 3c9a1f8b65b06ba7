"""The FP64 collisions inside and outside the range of the integer pipe
(mglc_gb300/csrc/fix61.cuh) against the oracle: cells of either kind side by
side, on rows that do not fill a warp.  Bound: the oracle rounds each of its
moment sums (the energy moment reaches 30 f, 19 terms) and divides by constants,
about 30 roundings of values up to 30 max|f| in one step: 30 * 30 * 2^-53, twice
that for two steps."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
EX = np.array([0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0])
EY = np.array([0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 0, 0, 0, 0, 1, -1, 1, -1])
EZ = np.array([0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1])
W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


@pytest.fixture(scope="module")
def mg():
    from mglc_gb300 import build
    build.build()
    import mglc_gb300
    return mglc_gb300


def _state(kind, shape, seed):
    """(nz, ny, nx, 19) populations near equilibrium; the kinds other than
    "flow" leave the integer range."""
    rng = np.random.default_rng(seed)
    kinds = ("flow", "dense", "thin", "fast", "edge")
    pick = np.full(shape, kinds.index(kind)) if kind != "mixed" else rng.integers(0, 5, shape)
    rho = np.choose(pick, [1.0, 4.0, 0.05, 1.0, 2.0]) * (1 + 0.02 * (rng.random(shape) - 0.5))
    u = (rng.random((3, *shape)) - 0.5) * np.choose(pick, [0.2, 0.1, 0.1, 0.9, 0.1])
    un = EX * u[0][..., None] + EY * u[1][..., None] + EZ * u[2][..., None]
    f = rho[..., None] * W * (1 + 3 * un + 4.5 * un * un - 1.5 * (u * u).sum(0)[..., None])
    return f * (1 + 0.01 * (rng.random(f.shape) - 0.5))


def _macros(f, force=0.0):
    rho = f.sum(-1)
    return rho, (f @ EX) / rho, (f @ EY) / rho, (f @ EZ) / rho


def _close(got, want, steps):
    bound = steps * 30 * 30 * 2.0 ** -53 * np.abs(want).max()
    assert np.abs(got - want).max() <= bound


@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("macros", [False, True])
@pytest.mark.parametrize("kind", ["flow", "dense", "thin", "fast", "edge", "mixed"])
def test_lid_matches_oracle_in_and_out_of_range(mg, kind, macros, in_place):
    nx, ny, nz = 33, 5, 4
    f = _state(kind, (nz, ny, nx), 3)
    m = _macros(f)
    if macros:  # a first step whose macro arrays do not agree with the populations
        m = (np.full_like(m[0], 1.0), 0.5 * m[1], 0.5 * m[2], 0.5 * m[3])
    o = O.LidOracle(nx, ny, nz, 300.0, 0.1)
    o.s.f[:] = f
    o.s.rho[:], o.s.u[:], o.s.v[:], o.s.w[:] = m
    with mg.LidDrivenCavity(nx, ny, nz, reynolds=300.0, u0=0.1, in_place=in_place) as c:
        c.load_state(f, *m) if macros else c.load_state(f)
        for n in (1, 2):
            c.step(1)
            o.run(1)
            _close(c.get_f(), o.s.f, n)


@pytest.mark.parametrize("reynolds", [0.5, 1e6])
def test_lid_matches_oracle_over_relaxation_times(mg, reynolds):
    """tau = 20 and 0.5 + 1e-5: both ends of the relaxation rates."""
    nx, ny, nz = 34, 4, 5
    f = _state("flow", (nz, ny, nx), 5)
    o = O.LidOracle(nx, ny, nz, reynolds, 0.1)
    o.s.f[:] = f
    o.s.rho[:], o.s.u[:], o.s.v[:], o.s.w[:] = _macros(f)
    with mg.LidDrivenCavity(nx, ny, nz, reynolds=reynolds, u0=0.1) as c:
        c.load_state(f)
        c.step(2)
        o.run(2)
        _close(c.get_f(), o.s.f, 2)


@pytest.mark.parametrize("ekman", [0.0, 1e-3])
@pytest.mark.parametrize("macros", [False, True])
@pytest.mark.parametrize("kind", ["flow", "dense", "fast", "edge", "mixed"])
def test_heated_matches_oracle_in_and_out_of_range(mg, kind, macros, ekman):
    nx, ny, nz = 33, 6, 5
    ra = 1e5
    f = _state(kind, (nz, ny, nx), 9)
    rng = np.random.default_rng(10)
    m = _macros(f)
    o = O.ThermalOracle(nx, ny, nz, ra, 0.71, 0.1, ekman, 0.5, -0.5, 0.0)
    T = rng.random((nz, ny, nx)) - 0.5
    g = T[..., None] * (np.array([0.4] + [0.1] * 6) * (1 + 0.02 * (rng.random((nz, ny, nx, 7)) - 0.5)))
    T = g.sum(-1)
    if macros:
        m, T = (np.full_like(m[0], 1.0), 0.5 * m[1], 0.5 * m[2], 0.5 * m[3]), 0.9 * T
    o.f[:], o.g[:], o.T[:] = f, g, T
    o.rho[:], o.u[:], o.v[:], o.w[:] = m
    with mg.BuoyancyCavity(nx, ny, nz, rayleigh=ra, prandtl=0.71, mach=0.1, t_hot=0.5, t_cold=-0.5,
                           ekman=ekman) as c:
        c.load_state(f, g, *m, T) if macros else c.load_state(f, g)
        for n in (1, 2):
            c.step(1)
            o.run(1)
            gf, gg = c.get_f()
            _close(gf, o.f, n)
            _close(gg, o.g, n)


def test_non_finite_cells_stay_non_finite(mg):
    """A NaN and an infinity take the FP64 form and spread with the stream, as in FP64."""
    f = _state("flow", (6, 6, 34), 7)
    f[2, 2, 5, 3], f[4, 3, 20, 0] = np.nan, np.inf
    with mg.LidDrivenCavity(34, 6, 6, reynolds=300.0, u0=0.1) as c:
        c.load_state(f)
        c.step(1)
        g = c.get_f()
    assert np.isnan(g).sum() == 38 and np.isfinite(g[0, 0, 0]).all()
