"""The status of a failed step: a kernel whose blocks meet at barriers reads it once for
the whole block (another block of the same launch may be setting it), and many
particles failing in one step freeze the state that they started the step with."""
import os
import re

import numpy as np
import pytest

from tests.test_particle_gpu import CASE, mg  # noqa: F401  (fixture)

CSRC = os.path.join(os.path.dirname(__file__), "..", "mglc_gb300", "csrc")


def _kernels(src):
    """name -> body of every kernel in src"""
    out = {}
    for m in re.finditer(r"__global__[^;{]*?\b(k2?_\w+)\s*\(", src):
        i = src.index("{", m.end())
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            j += 1
        out[m.group(1)] = src[i:j]
    return out


@pytest.mark.parametrize("name", ["k_particle.cu", "k_particle2d.cu"])
def test_blocks_with_barriers_leave_together(name):
    kernels = _kernels(open(os.path.join(CSRC, name)).read())
    assert len(kernels) > 8
    seen = 0
    for kernel, body in kernels.items():
        if "__syncthreads()" not in body and "block_sum_to<" not in body:
            continue
        lone = re.findall(r"if \([^;{]*(?:d\.status\[0\]|fetch\.stop\(\))\)*\s*return;", body)
        assert all("__syncthreads_or(" in x for x in lone), (kernel, lone)
        seen += bool(re.search(r"stopped\(d\)\)|__syncthreads_or\((?:fetch\.stop\(\)|code)", body))
    assert seen >= 3


def _grid(n, pitch, first):
    return [[first + pitch * i, first + pitch * j] for j in range(n) for i in range(n)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_many_spheres_failing_at_once_freeze_the_start(mg, precision):  # noqa: F811
    """Pairs closer than two radii, 96 of them, in the first step."""
    kw = dict(CASE)
    r = kw.pop("radius")
    for k in ("nx", "ny", "nz"):
        kw.pop(k)
    kw["periodic_x"] = bool(kw["periodic_x"])
    c3 = [[x, y, z] for x in np.arange(6.5, 190, 7.7) for y in (7.0, 13.5) for z in (8.0, 14.6, 21.0, 27.5)]
    for _ in range(3):
        with mg.ParticleFlow(192, 21, 36, c3, r, precision=precision, **kw) as c:
            c.initial()
            before = c.mask()
            with pytest.raises(mg.MglcError) as e:
                c.step(3)
            assert e.value.code == 7
            st = c.state()
            assert np.array_equal(c.mask(), before)
            assert np.array_equal(st["xc"], np.array(c3)) and not st["uc"].any()
            with pytest.raises(mg.MglcError):
                c.step(1)
            assert np.array_equal(c.state()["xc"], np.array(c3))


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [2.2, 3.6])
def test_many_circles_failing_at_once_freeze_the_start(mg, radius):  # noqa: F811
    """A 16x16 grid of circles closer than two radii."""
    centers = np.array(_grid(16, 2 * radius - 0.3, radius + 2.5))
    n = int(centers.max() + radius + 3)
    for _ in range(3):
        with mg.ParticleFlow2D(n, n, centers, radius) as c:
            c.initial()
            before = c.mask()
            with pytest.raises(mg.MglcError) as e:
                c.step(3)
            assert e.value.code == 7
            st = c.state()
            assert np.array_equal(st["xc"][:, :2], centers) and not st["uc"].any()
            assert np.array_equal(c.mask(), before)
            c.initial()  # and starts over
            with pytest.raises(mg.MglcError):
                c.step(1)
            assert np.array_equal(c.state()["xc"][:, :2], centers)
