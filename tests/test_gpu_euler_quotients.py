"""The reciprocals and quotients of csrc/euler_march.cuh are the correctly rounded
ones: over 1e9 pairs of their safe ranges (mantissas of all ones and their
neighbours, powers of two, quotients a few ulps from a midpoint, the ranges' ends)
none differs from CUDA's __drcp_rn and __ddiv_rn (tests/device/quotients.cu)."""
import os
import subprocess

import pytest

from test_host_layout import HERE, _nvcc

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_quotients_are_correctly_rounded(tmp_path):
    exe = str(tmp_path / "quotients")
    src = os.path.join(HERE, "device", "quotients.cu")
    r = subprocess.run([_nvcc(), "-O3", "--fmad=false", "-std=c++17", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-o", exe, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    pairs, *wrong = (int(x) for x in r.stdout.split())
    assert pairs > 10 ** 9 and wrong == [0, 0, 0]
