"""Euler's routes besides its default one.  threads=256: the shared-memory prisms
and seams (swept) and the per-cell kernel (standard).  Constants for which the
marching warps' quotients have no proven range (gamma - 1 next to zero, steps next
to nothing): the marching warps by plain divisions, alone and batched.  All equal
the per-cell kernel bitwise, and the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _ic(nx, ny):
    from pysweep_b200.equations.euler import analytical_array
    return analytical_array(nx, ny, 0.0)


def _globals(n):
    dx = 10.0 / n
    return [0.0, 1.0, 0.1 * dx, dx, dx, 1.4]


def _solve(ic, nl, bs, mode, consts=(), gts0=1, frames=False, kinds=None, **cfg):
    from pysweep_b200 import Engine, plugin_constants
    _, nx, ny = ic.shape
    with Engine("euler", nx, ny, its=2, blocksize=bs) as e:
        for k, v in {**plugin_constants("euler", _globals(nx)), **dict(consts)}.items():
            e.set_global(k, v)
        e.configure(**cfg)
        e.set_state(ic)
        e.profile(kinds is not None)
        fr = np.empty((nl // 2,) + ic.shape) if frames else None
        e.run(nl, mode=mode, gts0=gts0, frames=fr)
        if kinds is not None:
            kinds.update({k: v[1] for k, v in e.profile_read().items() if v[1]})
        return (e.get_state(0), e.get_state(1)) + ((fr,) if frames else ())


def _same(a, b):
    return all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


@pytest.mark.parametrize("bs,cfg", [(16, {}), (16, {"chunk": 32}), (16, {"chunk": 32, "nseg": 4}), (32, {}),
                                    (12, {"chunk": 32}), (8, {}), (16, {"h": 2}), (32, {"nseg": 2, "h": 5})])
@pytest.mark.parametrize("nl,gts0", [(14, 1), (9, 2)])
def test_prisms_match_march_and_per_cell_step(bs, cfg, nl, gts0):
    n = 96 if bs == 12 else (64 if bs == 8 else 128)
    ic = _ic(n, n)
    kinds = {}
    prism = _solve(ic, nl, bs, "swept", gts0=gts0, frames=True, kinds=kinds, threads=256, **cfg)
    assert {"prism", "ybridge", "gap", "octahedron"} <= set(kinds)
    march = _solve(ic, nl, bs, "swept", gts0=gts0, frames=True, **{k: v for k, v in cfg.items() if k == "h"})
    cell = _solve(ic, nl, bs, "standard", gts0=gts0, frames=True, threads=256)
    assert _same(prism, march) and _same(prism, cell)
    frames, last, older = oracle.standard("euler", ic, _globals(n), 2, nl, gts0=gts0, euler_square="mul")
    assert np.array_equal(prism[0], last) and np.array_equal(prism[1], older)
    if gts0 == 1:  # (the oracle's frames count from globalTimeStep, a run's from its start)
        assert np.array_equal(prism[2], frames[1:])


OUTSIDE = [{"GAM_M1": 2.0 ** -21}, {"GAM_M1": 0.0}, {"DTDX": 2.0 ** -1000}, {"DTDY": 1e-320},
           {"GAMMA": 2.0 ** 21, "GAM_M1": 0.4}]


@pytest.mark.parametrize("consts", OUTSIDE, ids=[",".join(c) + str(i) for i, c in enumerate(OUTSIDE)])
@pytest.mark.parametrize("mode", ["swept", "standard"])
def test_constants_outside_the_proven_ranges(consts, mode):
    for nx, ny, bs, nl, gts0 in ((64, 120, 8, 7, 1), (96, 64, 16, 6, 2)):
        ic = _ic(nx, ny)
        kinds = {}
        got = _solve(ic, nl, bs, mode, consts, gts0, kinds=kinds)
        assert kinds == {"block" if mode == "swept" else "standard": nl}  # one launch per level
        assert _same(got, _solve(ic, nl, bs, "standard", consts, gts0, threads=256))


@pytest.mark.parametrize("graph", [True, False])
def test_batch_with_constants_outside_the_proven_ranges(graph):
    """Instances inside and outside, in one batch."""
    from pysweep_b200 import Batch, plugin_constants
    sizes = [(32, 64), (64, 96), (48, 128), (64, 16), (16, 16), (80, 64)]
    with Batch("euler", sizes, its=2, blocksize=16) as b:
        for i, s in enumerate(sizes):
            b.set_constants(i, {**plugin_constants("euler", _globals(s[0])), **([{}] + OUTSIDE)[i]})
            b.set_state(i, _ic(*s))
        b.run(5, graph=graph)
        b.run(4, graph=graph)
        got = [(b.get_state(i, 0), b.get_state(i, 1)) for i in range(len(sizes))]
    for i, s in enumerate(sizes):
        assert _same(got[i], _solve(_ic(*s), 9, 16, "standard", ([{}] + OUTSIDE)[i], threads=256))
