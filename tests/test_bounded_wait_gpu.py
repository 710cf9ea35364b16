"""The bounded wait on an mbarrier (csrc/common.cuh) that the PP and PM3 kernels use: all lanes of a warp get one
answer, also where the barrier completes between the limits of two lanes, and a wait that runs out returns."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
MS = 1_000_000


@pytest.fixture(scope="module")
def probe(gpu, tmp_path_factory):
    from cube2_b200 import build as B
    so = str(tmp_path_factory.mktemp("probe") / "libwait_probe.so")
    subprocess.run([B.NVCC, *B.ARCH, *B.FLAGS, "-I", B.CSRC, "-shared", os.path.join(HERE, "wait_probe.cu"), "-o", so],
                   check=True)
    fn = ctypes.CDLL(so).wait_probe
    fn.argtypes = [ctypes.c_ulonglong] * 3 + [ctypes.POINTER(ctypes.c_int)]

    def run(limit, step, arrive):
        ok = (ctypes.c_int * 32)()
        assert fn(limit, step, arrive, ok) == 0
        return list(ok)
    return run


def test_all_lanes_get_one_answer(probe):
    # complete well within every limit; never; and (lane limits 0.2 to 6.4 ms) after some lanes' limits and before others'
    assert probe(1000 * MS, 0, MS // 5) == [1] * 32
    assert probe(2 * MS, 0, 0) == [0] * 32
    assert probe(MS // 5, MS // 5, 3 * MS) == [0] * 32
