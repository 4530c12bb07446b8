"""The standard decomposition's heat kernel (csrc/standard_fast.cuh) where its
strips of 64 columns and four or eight rows end: single blocks, rows that are no
multiple of 64 columns or of eight rows, both schemes beginning with either stage,
odd level counts, forward Euler with two base levels, frames at any address.
Bitwise against the oracle's level-by-level stepper (the same operations in the
same order)."""
import numpy as np
import pytest

import oracle
from test_gpu_block import _globals, _ic, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,bs", [(8, 8, 8), (12, 60, 12), (9 * 4, 64, 4), (66, 66, 6), (40, 130, 10),
                                      (1120, 1120, 16), (2048, 2112, 32)])
@pytest.mark.parametrize("its,euler,gts0,nl", [(1, True, 1, 3), (2, False, 1, 5), (2, False, 2, 4),
                                               (2, True, 1, 3)])
def test_standard_rows(nx, ny, bs, its, euler, gts0, nl):
    ic, g = _ic(nx, ny), _globals(nx, euler)
    got, _ = _solve(ic, g, its, bs, nl, mode="standard", gts0=gts0)
    _, ref, refp = oracle.standard("heat", ic, g, its, nl, gts0=gts0, frames=False)
    assert np.array_equal(got[0], ref)
    if its == 2:
        assert np.array_equal(got[1], refp)


@pytest.mark.parametrize("nx,ny", [(16, 64), (50 * 2, 128)])
def test_standard_rows_float32(nx, ny):
    ic, g = _ic(nx, ny).astype(np.float32), _globals(nx)
    (u,), _ = _solve(ic, g, 1, 4, 5, mode="standard", dtype="float32")
    assert np.array_equal(u, oracle.heat_f32(ic, g, 5))


@pytest.mark.parametrize("its,off", [(1, 0), (1, 1), (2, 0), (2, 1)])
def test_standard_rows_frames(its, off):
    import torch
    from pysweep_b200 import Engine, plugin_constants
    nx, ny, nl = 36, 66, 6
    ic, g = _ic(nx, ny), _globals(nx, its == 1)
    flat = torch.zeros(off + nl // its * nx * ny, dtype=torch.float64, device="cuda")
    fr = flat[off:].view(-1, 1, nx, ny)
    with Engine("heat", nx, ny, its=its, blocksize=6) as e:
        for k, v in plugin_constants("heat", g).items():
            e.set_global(k, v)
        e.set_state(ic)
        e.run(nl, mode="standard", frames=fr)
        e.synchronize()
    ref, _, _ = oracle.standard("heat", ic, g, its, nl)
    assert np.array_equal(fr.cpu().numpy(), ref[1:])
