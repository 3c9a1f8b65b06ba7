"""Macroscopic fields of the reduced forms (mglc_gb300/csrc/macro64.cuh): the integer
sums and the FP64 ones for what lies outside their range (a stored deviation of 1/8
or more), against extended-precision sums of the populations
themselves.  Bounds: a population read back is rounded at 2^-53 of its size (19 of
them, up to 4), the fields at 2^-53: 19 * 4 * 2^-53 on rho, twice that over rho on the
velocity."""
import numpy as np
import pytest

from tests.test_fix61_gpu import EX, EY, EZ, mg  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu
W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


def _state(kind, shape, q, rng):
    rho = 1.0 + 0.02 * (rng.random(shape) - 0.5)
    f = rho[..., None] * W * (1 + 0.1 * (rng.random((*shape, 19)) - 0.5))
    if kind == "rest":
        f[:] = W
    elif kind == "tiny":  # deviations down to 2^-60
        f = W * (1 + 2.0 ** -rng.integers(10, 52, (*shape, 19)))
    elif kind == "dense":  # rest deviations on either side of 1/8
        f = 1.375 * (1 + 0.02 * (rng.random(shape) - 0.5))[..., None] * W
    elif kind == "thin":
        f = 0.25 * (1 + 0.05 * (rng.random(shape) - 0.5))[..., None] * W
    return f


@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16", "fp16s"])
@pytest.mark.parametrize("kind", ["flow", "rest", "tiny", "dense", "thin"])
def test_fields_are_the_populations_sums(mg, precision, kind):  # noqa: F811
    nx, ny, nz = 35, 6, 5
    rng = np.random.default_rng(3)
    f = _state(kind, (nz, ny, nx), 19, rng)
    with mg.LidDrivenCavity(nx, ny, nz, reynolds=100.0, u0=0.05, precision=precision) as c:
        c.load_state(f)
        c.step(1)
        rho, u, v, w = c.macro()[:4]
        g = c.get_f().astype(np.longdouble)
    r = g.sum(-1)
    tol = 19 * 4 * 2.0 ** -53
    assert np.abs(rho - r).max() <= tol
    for got, e in ((u, EX), (v, EY), (w, EZ)):
        assert (np.abs(got - (g * e).sum(-1) / r) * np.abs(r)).max() <= 2 * tol


@pytest.mark.parametrize("precision", ["fp32", "fp16s"])
def test_heated_fields(mg, precision):  # noqa: F811
    """Temperatures on either side of the integer sum's range (populations below 1)."""
    nx, ny, nz = 33, 5, 6
    rng = np.random.default_rng(4)
    f = _state("flow", (nz, ny, nx), 19, rng)
    T = np.where(rng.random((nz, ny, nx)) < 0.5, 1.0, 4.0) * (rng.random((nz, ny, nx)) - 0.5)
    g = T[..., None] * (np.array([0.4] + [0.1] * 6))
    g[0, 0, :5] = 1.5
    with mg.BuoyancyCavity(nx, ny, nz, rayleigh=1e4, t_hot=0.5, t_cold=-0.5, precision=precision) as c:
        c.load_state(f, g)
        c.step(1)
        fields = c.macro()
        fg = c.get_f()
    f2, g2 = fg
    f2, g2 = f2.astype(np.longdouble), g2.astype(np.longdouble)
    r = f2.sum(-1)
    tol = 19 * 4 * 2.0 ** -53
    assert np.abs(fields[0] - r).max() <= tol
    for got, e in ((fields[1], EX), (fields[2], EY)):  # no force in x and y
        assert (np.abs(got - (f2 * e).sum(-1) / r) * np.abs(r)).max() <= 2 * tol
    assert np.abs(fields[4] - g2.sum(-1)).max() <= 7 * 4 * 2.0 ** -53


@pytest.mark.parametrize("precision", ["fp32", "fp16s"])
@pytest.mark.parametrize("scale", [0.0, 1e-16, 1e-11, 1e-6, 1.0, 300.0, 1e-30])
def test_temperature_of_any_scale(mg, scale, precision):  # noqa: F811
    """Bound: seven units of 2^-59 of the largest population, and the rounding of the sum."""
    nx, ny, nz = 33, 5, 6
    rng = np.random.default_rng(4)
    f = _state("flow", (nz, ny, nx), 19, rng)
    T = scale * (rng.random((nz, ny, nx)) - 0.5)
    g = T[..., None] * (np.array([0.4] + [0.1] * 6)) * (1 + 0.1 * rng.random((nz, ny, nx, 7)))
    with mg.BuoyancyCavity(nx, ny, nz, rayleigh=1e4, t_hot=0.5 * scale, t_cold=-0.5 * scale, precision=precision) as c:
        c.load_state(f, g)
        c.step(1)
        got = c.macro()[4]
        g2 = c.get_f()[1].astype(np.longdouble)
    want = g2.sum(-1)
    assert np.isfinite(got).all()
    assert (np.abs(got - want) <= 7 * 2.0 ** -59 * np.abs(g2).max(-1) + 8 * 2.0 ** -53 * np.abs(g2).sum(-1)).all()
