"""Steps whose launches overlap the kernel before (mglc_gb300/csrc/launch.cuh): the
same bits from one call, from single calls with the fields read in between, on a
stream of the caller's and replayed from a captured graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mg():
    from mglc_gb300 import build
    build.build()
    import mglc_gb300
    return mglc_gb300


def _make(mg, kind, in_place):
    if kind == "lid":
        return mg.LidDrivenCavity(33, 17, 9, reynolds=100.0, u0=0.1, precision="fp32", in_place=in_place)
    return mg.BuoyancyCavity(32, 9, 17, rayleigh=1e4, t_hot=0.5, t_cold=-0.5, in_place=in_place)


@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("kind", ["lid", "heated"])
def test_steps_are_serial(mg, kind, in_place):
    import torch
    f = {}
    with _make(mg, kind, in_place) as c:
        c.initial()
        c.step(7)
        f["one call"] = c.get_f()
    with _make(mg, kind, in_place) as c:
        c.initial()
        for _ in range(7):
            c.step(1)
            c.macro()
        f["single"] = c.get_f()
    s = torch.cuda.Stream()
    with _make(mg, kind, in_place) as c:
        c.set_stream(s.cuda_stream)
        c.initial()
        c.step(1)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            c.step(2)
        for _ in range(3):
            g.replay()
        torch.cuda.synchronize()
        f["graph"] = c.get_f()
    ref = f["one call"]
    for k, v in f.items():
        for a, b in zip(ref if isinstance(ref, tuple) else (ref,), v if isinstance(v, tuple) else (v,)):
            assert np.array_equal(a, b), k
