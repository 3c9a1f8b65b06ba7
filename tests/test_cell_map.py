"""Cells by thread index (mglc_gb300/csrc/cell_map.cuh): the division by
multiplication, and ragged grids against the oracle on the linear order
(tests/test_fix61_gpu.py and test_edges_gpu.py cover the rows)."""
import random

import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_util import rel_l2


def _div(d):
    sh = 1
    while (1 << sh) < d:
        sh += 1
    m = (1 << (31 + sh)) // d + 1
    assert m < 1 << 32
    return m, sh - 1


def test_division_by_multiplication():
    rng = random.Random(5)
    for d in list(range(2, 700)) + [rng.randrange(2, 1 << 27) for _ in range(400)] + [1 << k for k in range(1, 28)]:
        m, s = _div(d)
        ns = [0, 1, d - 1, d, d + 1, (1 << 31) - 1] + [rng.randrange(1 << 31) for _ in range(20)]
        top = ((1 << 31) - 1) // d
        ns += [q * d + e for q in (1, 2, top // 2, top - 1, top) for e in (-1, 0) if q >= 1]
        for n in ns:
            if 0 <= n < 1 << 31:
                assert (n * m >> 32) >> s == n // d, (n, d)


@pytest.fixture(scope="module")
def mg():
    from mglc_gb300 import build
    build.build()
    import mglc_gb300
    return mglc_gb300


@pytest.mark.gpu
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("shape", [(2, 3, 2), (31, 5, 3), (33, 2, 7), (65, 4, 3), (129, 3, 2), (160, 2, 3)])
def test_ragged_rows_match_oracle(mg, shape, in_place):
    """FP64 1e-12, FP32 2e-6 of the largest population (the bounds of the step
    kernels' tests over few steps)."""
    nx, ny, nz = shape
    o = O.LidOracle(nx, ny, nz, 200.0, 0.1)
    o.run(6)
    for precision, tol in (("fp64", 1e-12), ("fp32", 2e-6)):
        with mg.LidDrivenCavity(nx, ny, nz, reynolds=200.0, u0=0.1, precision=precision, in_place=in_place) as c:
            c.initial()
            c.step(6)
            assert rel_l2(c.get_f(), o.s.f) <= tol
