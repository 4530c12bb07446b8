"""Step hooks in overlapped blocks (csrc/hook_kernels.cuh, psh_block) where tiles
and launches end: grids smaller than a tile, one cell over it, level counts around
a launch's, frames, one and two base levels, wide stencils and many variables (one
level per launch).  Bitwise against the oracle for heat; for the two-variable
five-point system and a many-variable stencil, against the shared-memory prisms
(threads=256), which run the same compiled hook."""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
HOOKS = os.path.join(os.path.dirname(os.path.abspath(__file__)), "hooks")

# nv variables, a stencil of reach OPS: each variable from the next one's
# neighbours at every distance
MANY = """
__device__ void step(double *s, int idx, int globalTimeStep)
{
    for (int v = 0; v < NV; ++v) {
        const int q = idx + v * VARS, w = idx + (v + 1) % NV * VARS;
        double a = 0;
        for (int k = 1; k <= OPS; ++k)
            a += (s[w + k * SY] - s[w - k * SY]) / (k + 1) + (s[w + k] + s[w - k]) / (k + 2);
        s[q + TIMES] = 0.5 * s[q] + 0.05 * a;
    }
}
"""


def _run(ic, levels, bs, mode="swept", its=1, ops=1, path=None, source=None, consts=(), every=0,
         gts0=1, **cfg):
    from pysweep_b200 import Engine
    nv, nx, ny = ic.shape
    with Engine(path or "many", nx, ny, nv=nv, ops=ops, its=its, blocksize=bs, hook_source=source) as e:
        for k, v in dict(consts).items():
            e.set_global(k, v)
        e.configure(**cfg)
        e.set_state(ic)
        fr = np.empty((levels // its // every,) + ic.shape) if every else None
        e.run(levels, mode=mode, gts0=gts0, frames=fr, frame_every=every or 1)
        return [e.get_state(q) for q in range(its)], fr


def _heat(n, euler):
    from pysweep_b200 import plugin_constants
    g = [0.0, 1.0, 0.2 / n / n, 1 / n, 1 / n, 1.0, euler]
    return g, plugin_constants("heat", g)


@pytest.mark.parametrize("nx,ny,bs", [(8, 8, 8), (24, 60, 6), (28, 60, 4), (32, 64, 16), (56, 120, 8)])
@pytest.mark.parametrize("its,nl", [(1, 1), (1, 4), (1, 9), (2, 4), (2, 11)])
def test_heat_hook_blocks(nx, ny, bs, its, nl):
    ic = np.random.default_rng([nx, ny]).standard_normal((1, nx, ny))
    g, consts = _heat(nx, its == 1)
    every = 1 if nl >= 2 * its else 0
    got, fr = _run(ic, nl, bs, its=its, path=os.path.join(HOOKS, "heat_numpy_order.cu"), consts=consts,
                   every=every)
    ref, last, prev = oracle.standard("heat", ic, g, its, nl)
    assert np.array_equal(got[0], last) and (its == 1 or np.array_equal(got[1], prev))
    if every:
        assert np.array_equal(fr, ref[1:])


@pytest.mark.parametrize("nx,ny,bs", [(16, 16, 16), (32, 64, 16), (48, 80, 16)])
@pytest.mark.parametrize("nl,gts0", [(1, 1), (7, 2), (10, 1)])
def test_two_variable_hook_blocks(nx, ny, bs, nl, gts0):
    ic = np.random.default_rng([nx, ny, nl]).standard_normal((2, nx, ny))
    kw = dict(its=2, ops=2, path=os.path.join(HOOKS, "wave4.cu"), consts={"A": 0.7, "DT": 0.05}, gts0=gts0)
    got, _ = _run(ic, nl, bs, **kw)
    ref, _ = _run(ic, nl, bs, threads=256, **kw)
    std, _ = _run(ic, nl, bs, mode="standard", **kw)
    for a, b, c in zip(got, ref, std):
        assert np.array_equal(a, b) and np.array_equal(a, c)


@pytest.mark.parametrize("nv,ops", [(1, 1), (2, 1), (3, 1), (1, 2), (1, 4), (4, 2), (8, 4)])
def test_shapes_of_hooks(nv, ops):
    nx, ny, bs, nl = 40, 80, 4 * ops if ops > 1 else 8, 5
    nx, ny = nx - nx % bs + bs, ny - ny % bs + bs
    ic = np.random.default_rng([nv, ops]).standard_normal((nv, nx, ny))
    got, _ = _run(ic, nl, bs, ops=ops, source=MANY)
    std, _ = _run(ic, nl, bs, ops=ops, source=MANY, mode="standard")
    assert np.array_equal(got[0], std[0])
    ref = ic
    for _ in range(nl):  # the hook on whole arrays, in its order
        w = np.roll(ref, -1, axis=0)
        a = np.zeros_like(ref)
        for k in range(1, ops + 1):
            a = a + ((np.roll(w, -k, 1) - np.roll(w, k, 1)) / (k + 1) +
                     (np.roll(w, -k, 2) + np.roll(w, k, 2)) / (k + 2))
        ref = 0.5 * ref + 0.05 * a
    assert np.array_equal(got[0], ref)
