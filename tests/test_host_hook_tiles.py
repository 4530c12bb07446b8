"""The step hooks' tiles for every number of variables and reach, compiled with
nvcc and run on the CPU (tests/host/hook_tiles.cu)."""
import os
import subprocess

import pytest

from test_host_layout import HERE, _nvcc


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_hook_tiles(tmp_path):
    exe = str(tmp_path / "hook_tiles")
    src = os.path.join(HERE, "host", "hook_tiles.cu")
    r = subprocess.run([_nvcc(), "-std=c++17", "-arch=sm_100a", "-o", exe, src, "-ldl"], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
