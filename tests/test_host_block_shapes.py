"""The grids of test_gpu_block_shapes.py take every tile that is built, and the
streams: a plan refitted so that a kernel drops out of test fails here
(tests/host/block_shapes.cu, compiled with nvcc and run on the CPU)."""
import os
import subprocess

import pytest

from block_grids import GRIDS
from test_host_layout import HERE, _nvcc


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_every_shape_is_planned(tmp_path):
    exe = str(tmp_path / "block_shapes")
    src = os.path.join(HERE, "host", "block_shapes.cu")
    r = subprocess.run([_nvcc(), "-std=c++17", "-arch=sm_100a", "-o", exe, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def ask(lines):
        r = subprocess.run([exe], input="".join(f"{a} {b} {c} {d}\n" for a, b, c, d in lines),
                           capture_output=True, text=True)
        assert r.returncode == 0
        return [set(x.split()) for x in r.stdout.splitlines()]

    for kind, grids in GRIDS.items():
        built, = ask([(kind, 0, 0, 0)])
        taken = set().union(*ask([(kind, *g) for g in grids]))
        assert taken == built, kind
