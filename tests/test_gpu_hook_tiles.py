"""Step hooks, one level per launch, in every tile that numbers of variables and
reaches lead to (hook_block in csrc/hook.cuh): grids smaller than a tile, one row
and two columns over one, whole tiles.  Bitwise against the hook on whole arrays."""
import numpy as np
import pytest

from test_gpu_hook_block import MANY, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv,ops", [(1, 1), (1, 2), (2, 1), (3, 1), (3, 2), (4, 4), (5, 3), (6, 2), (7, 4), (8, 1),
                                    (8, 4)])
@pytest.mark.parametrize("nx,ny", [(24, 24), (48, 144), (72, 72)])
@pytest.mark.parametrize("its", [1, 2])
def test_standard_hook_tiles(nv, ops, nx, ny, its):
    bs = 4 * ops
    nx, ny = -(-nx // bs) * bs, -(-ny // bs) * bs
    ic = np.random.default_rng([nv, ops, nx]).standard_normal((nv, nx, ny))
    nl = 3
    got, _ = _run(ic, nl, bs, ops=ops, its=its, source=MANY, mode="standard")
    new = ic
    for _ in range(nl):
        old, w = new, np.roll(new, -1, axis=0)
        a = np.zeros_like(old)
        for k in range(1, ops + 1):
            a = a + ((np.roll(w, -k, 1) - np.roll(w, k, 1)) / (k + 1) +
                     (np.roll(w, -k, 2) + np.roll(w, k, 2)) / (k + 2))
        new = 0.5 * old + 0.05 * a
    assert np.array_equal(got[0], new) and (its == 1 or np.array_equal(got[1], old))
