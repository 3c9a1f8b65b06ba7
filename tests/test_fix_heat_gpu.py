"""Temperature populations of the FP64 heated cavity on the integer pipe
(mglc_gb300/csrc/fix61.cuh, fix_heat) and, a population of 1/2 or a temperature of 1
or more, in FP64: against the oracle, cells of either kind side by side.  Bound a
step: the oracle's own rounding (test_fix61_gpu.py: 30 * 30 * 2^-53 of the largest
value) and eight units of 2^-61 for the loading and products of a population."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_fix61_gpu import _state, mg  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def _temperature(kind, shape, rng):
    T = rng.random(shape) - 0.5
    if kind == "zero":
        T[:] = 0.0
    elif kind == "tiny":  # down to far below 2^-61
        T *= 2.0 ** -rng.integers(0, 90, shape)
    elif kind == "hot":  # populations on either side of 1/2, temperatures of 1
        T *= np.where(rng.random(shape) < 0.5, 2.0, 2.6)
    return T


@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("ekman", [0.0, 1e-3])
@pytest.mark.parametrize("kind", ["plain", "zero", "tiny", "hot"])
def test_temperature_matches_oracle(mg, kind, ekman, in_place):  # noqa: F811
    nx, ny, nz = 35, 5, 6
    rng = np.random.default_rng(21)
    f = _state("flow", (nz, ny, nx), 8)
    T = _temperature(kind, (nz, ny, nx), rng)
    g = T[..., None] * (np.array([0.4] + [0.1] * 6))
    rho = f.sum(-1)
    o = O.ThermalOracle(nx, ny, nz, 1e5, 0.71, 0.1, ekman, 0.5, -0.5, 0.0)
    from tests.test_fix61_gpu import _macros
    m = _macros(f)
    T = g.sum(-1)
    o.f[:], o.g[:], o.T[:], o.rho[:] = f, g, T, rho
    o.u[:], o.v[:], o.w[:] = m[1:]
    with mg.BuoyancyCavity(nx, ny, nz, rayleigh=1e5, prandtl=0.71, mach=0.1, t_hot=0.5, t_cold=-0.5,
                           ekman=ekman, in_place=in_place) as c:
        c.load_state(f, g)
        for n in (1, 2, 3, 4):
            c.step(1)
            o.run(1)
            gf, gg = c.get_f()
            for got, want in ((gf, o.f), (gg, o.g)):
                bound = n * (900 * 2.0 ** -53 * np.abs(want).max() + 8 * 2.0 ** -61)
                assert np.abs(got - want).max() <= bound


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_cells_spread_as_in_the_oracle(mg, bad):  # noqa: F811
    """Cells whose density is not finite: not finite where the oracle is not (which of
    infinity and NaN a population becomes depends on the form of the sums), its
    values elsewhere."""
    nx, ny, nz = 34, 6, 7
    f = _state("flow", (nz, ny, nx), 8)
    T = 0.3 * np.sin(np.arange(nz * ny * nx)).reshape(nz, ny, nx)
    g = T[..., None] * (np.array([0.4] + [0.1] * 6))
    from tests.test_fix61_gpu import _macros
    m = _macros(f)
    f[3, 2, 16, 5] = bad
    o = O.ThermalOracle(nx, ny, nz, 1e5, 0.71, 0.1, 0.0, 0.5, -0.5, 0.0)
    o.f[:], o.g[:], o.T[:] = f, g, g.sum(-1)
    o.rho[:], o.u[:], o.v[:], o.w[:] = m
    with mg.BuoyancyCavity(nx, ny, nz, rayleigh=1e5, prandtl=0.71, mach=0.1, t_hot=0.5, t_cold=-0.5) as c, \
            np.errstate(all="ignore"):
        c.load_state(f, g, *m, g.sum(-1))
        for n in (1, 2, 3):
            c.step(1)
            o.run(1)
            for got, want in zip(c.get_f(), (o.f, o.g)):
                assert np.array_equal(np.isfinite(got), np.isfinite(want))
                ok = np.isfinite(want)
                bound = n * (900 * 2.0 ** -53 * np.abs(want[ok]).max() + 8 * 2.0 ** -61)
                assert np.abs(got[ok] - want[ok]).max() <= bound
