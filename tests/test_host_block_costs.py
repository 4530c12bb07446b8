"""The plans of two-stage, float32, per-cell-courant and backward launches and of
Euler's strips, compiled with nvcc and run on the CPU (tests/host/block_costs.cu)."""
import os
import subprocess

import pytest

from test_host_layout import HERE, _nvcc


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_plans_of_every_cost(tmp_path):
    exe = str(tmp_path / "block_costs")
    src = os.path.join(HERE, "host", "block_costs.cu")
    r = subprocess.run([_nvcc(), "-std=c++17", "-arch=sm_100a", "-o", exe, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
