"""How heat runs are cut into overlapped blocks, compiled with nvcc and run on
the CPU (tests/host/block_plan.cu)."""
import os
import subprocess

import pytest

from test_host_layout import HERE, _nvcc


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_block_plan(tmp_path):
    exe = str(tmp_path / "block_plan")
    src = os.path.join(HERE, "host", "block_plan.cu")
    r = subprocess.run([_nvcc(), "-std=c++17", "-arch=sm_100a", "-o", exe, src], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
