"""Kernels that are launched before the kernel before them has ended
(mglc_gb300/csrc/launch.cuh) read with plain loads: __ldg and const __restrict__ let the
compiler use the read-only path, which is for memory that nothing writes during the
kernel's lifetime."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "mglc_gb300", "csrc")


def _functions(src):
    """(signature, body) of every kernel"""
    for m in re.finditer(r"__global__", src):
        i = src.index("{", m.end())
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            j += 1
        yield src[m.start():i], src[i:j]


def test_overlapped_kernels_use_plain_loads():
    waiting = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        for sig, body in _functions(open(path).read()):
            if "after_previous();" not in body:
                continue
            waiting += 1
            assert body.split(";")[0].strip("{ \n") == "after_previous()", sig
            assert not re.search(r"const\s[^,()]*__restrict__", sig), sig
            assert "__ldg" not in body, sig
    assert waiting >= 20


def test_their_cell_bodies_too():
    for name in ("step_cell.cuh", "macro64.cuh", "fix61.cuh", "lbm_common.cuh", "d2q9.cuh"):
        src = open(os.path.join(CSRC, name)).read()
        assert not re.search(r"const\s[^,();]*__restrict__", src), name
        left = [x for x in src.splitlines() if "__ldg" in x]
        # St::ld, the server's fields and residual, launched the plain way
        assert all(re.search(r" C ld\(|return __bfloat162float\(__ldg\(p\)\) \* inv;", x) for x in left), left
    assert "__ldg" not in open(os.path.join(CSRC, "k_particle.cu")).read()
    assert "launch_next" not in open(os.path.join(CSRC, "k_serve.cu")).read()
