"""Heat through the overlapped blocks (csrc/heat_block.cuh) where a launch's
tiles and strips end: grids smaller than a tile, one column or row over a tile,
rows that are no multiple of four columns, level counts around a launch's, frames,
runs that begin with either stage.  Every field equals the oracle's level-by-level
stepper bitwise (the cell arithmetic is the same in every decomposition, so the
tolerance is zero); sizes too large for it, the per-cell standard kernel's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _solve(ic, g, its, bs, nl, mode="swept", gts0=1, every=0, dtype="float64", **cfg):
    from pysweep_b200 import Engine, plugin_constants
    _, nx, ny = ic.shape
    with Engine("heat", nx, ny, its=its, blocksize=bs, dtype=dtype) as e:
        for k, v in plugin_constants("heat", g).items():
            e.set_global(k, v)
        e.configure(**cfg)
        e.set_state(ic)
        fr = np.empty((nl // its // every,) + ic.shape, dtype=e.dtype) if every else None
        e.run(nl, mode=mode, gts0=gts0, frames=fr, frame_every=every or 1)
        return [e.get_state(q) for q in range(its)], fr


def _globals(n, euler=True):
    return [0.0, 1.0, 0.2 / n / n, 1 / n, 1 / n, 1.0, euler]


def _ic(nx, ny, seed=0):
    return np.random.default_rng([nx, ny, seed]).standard_normal((1, nx, ny))


@pytest.mark.parametrize("nx,ny,bs", [
    (8, 8, 8), (16, 136, 8), (48, 48, 16), (112, 112, 16), (120, 120, 8), (128, 224, 32),
    (330, 18, 6), (42, 390, 6), (80, 1120, 16), (560, 64, 16)])
@pytest.mark.parametrize("nl", [1, 7, 8, 9, 33])
def test_forward_euler_blocks(nx, ny, bs, nl):
    ic, g = _ic(nx, ny), _globals(nx)
    (u,), _ = _solve(ic, g, 1, bs, nl)
    _, ref, _ = oracle.standard("heat", ic, g, 1, nl, frames=False)
    assert np.array_equal(u, ref)


@pytest.mark.parametrize("nx,ny,bs", [(16, 16, 8), (64, 120, 8), (96, 390, 6), (128, 128, 32)])
@pytest.mark.parametrize("nl,gts0", [(1, 1), (2, 1), (2, 2), (7, 1), (8, 2), (21, 2), (34, 1)])
def test_two_stage_blocks(nx, ny, bs, nl, gts0):
    ic, g = _ic(nx, ny), _globals(nx, False)
    (u, up), _ = _solve(ic, g, 2, bs, nl, gts0=gts0)
    _, ref, refp = oracle.standard("heat", ic, g, 2, nl, gts0=gts0, frames=False)
    assert np.array_equal(u, ref) and np.array_equal(up, refp)


@pytest.mark.parametrize("nx,ny,bs,its,every", [(96, 120, 8, 1, 1), (96, 120, 8, 1, 5), (66, 90, 6, 1, 3),
                                                (64, 120, 8, 2, 1), (66, 90, 6, 2, 4)])
def test_block_frames(nx, ny, bs, its, every):
    nl = 23 * its
    ic, g = _ic(nx, ny), _globals(nx, its == 1)
    _, fr = _solve(ic, g, its, bs, nl, every=every)
    ref, _, _ = oracle.standard("heat", ic, g, its, nl)
    assert np.array_equal(fr, ref[every::every][: len(fr)])


@pytest.mark.parametrize("its,gts0", [(1, 1), (2, 1), (2, 2)])
def test_block_frames_at_any_address(its, gts0):
    """Device frames that start 8 bytes off a 32-byte boundary."""
    import torch
    from pysweep_b200 import Engine, plugin_constants
    nx, ny, nl = 64, 96, 20
    ic, g = _ic(nx, ny), _globals(nx, its == 1)
    out = []
    for off in (0, 1):
        flat = torch.zeros(off + nl // its * nx * ny, dtype=torch.float64, device="cuda")
        fr = flat[off:].view(-1, 1, nx, ny)
        with Engine("heat", nx, ny, its=its, blocksize=16) as e:
            for k, v in plugin_constants("heat", g).items():
                e.set_global(k, v)
            e.set_state(ic)
            e.run(nl, gts0=gts0, frames=fr)
            e.synchronize()
        out.append(fr.cpu().numpy())
    assert np.array_equal(out[0], out[1]) and np.abs(out[0]).sum() > 0


@pytest.mark.parametrize("nx,ny,bs,nl", [(32, 64, 16, 9), (128, 416, 32, 20)])
def test_float32_blocks(nx, ny, bs, nl):
    ic, g = _ic(nx, ny).astype(np.float32), _globals(nx)
    ic[0, 3, 5] = 1e-41  # a float32 subnormal
    (u,), _ = _solve(ic, g, 1, bs, nl, dtype="float32")
    assert np.array_equal(u, oracle.heat_f32(ic, g, nl))


@pytest.mark.parametrize("nx,ny,bs,its,nl", [
    (2048, 2048, 32, 1, 21), (1000, 4504, 8, 1, 16), (3000, 2000, 8, 2, 20), (2304, 2046, 6, 1, 8)])
def test_streams(nx, ny, bs, its, nl):
    """Grids the register streams take (the last: no multiple of four columns)."""
    ic, g = _ic(nx, ny), _globals(nx, its == 1)
    got, _ = _solve(ic, g, its, bs, nl)
    ref, _ = _solve(ic, g, its, bs, nl, mode="standard", threads=256)
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))


@pytest.mark.parametrize("nx,ny,bs,its,nl", [
    (1000, 1400, 8, 1, 23), (1280, 1280, 32, 1, 16), (1664, 1664, 32, 1, 25),
    (512, 512, 16, 2, 20), (702, 702, 6, 2, 17), (1000, 1400, 8, 2, 24), (1120, 1120, 16, 2, 9)])
def test_tiles_of_many_rows(nx, ny, bs, its, nl):
    """Grids whose plan takes the tiles of eight and ten rows per warp, alone and
    as a batch of one."""
    from pysweep_b200 import Batch, plugin_constants
    ic, g = _ic(nx, ny), _globals(nx, its == 1)
    got, _ = _solve(ic, g, its, bs, nl)
    ref, _ = _solve(ic, g, its, bs, nl, mode="standard", threads=256)
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))
    if its == 1 and nx % 32 == 0:
        with Batch("heat", [(nx, ny)], blocksize=bs) as b:
            b.set_constants(0, plugin_constants("heat", g))
            b.set_state(0, ic)
            b.run(nl)
            assert np.array_equal(b.get_state(0), ref[0])


@pytest.mark.parametrize("h", [1, 2, 5])
def test_configured_levels_bound_a_launch(h):
    nx, ny, nl = 96, 160, 11
    ic, g = _ic(nx, ny), _globals(nx)
    (u,), _ = _solve(ic, g, 1, 16, nl, h=h)
    _, ref, _ = oracle.standard("heat", ic, g, 1, nl, frames=False)
    assert np.array_equal(u, ref)


@pytest.mark.parametrize("sizes,runs", [
    ([(32, 32), (128, 480), (64, 160)], (5, 17)),          # tiles
    ([(2048, 2048), (64, 96), (32, 1056)], (20, 3)),       # streams, then tiles
])
@pytest.mark.parametrize("graph", [True, False])
def test_batched_blocks(sizes, runs, graph):
    from pysweep_b200 import Batch, plugin_constants
    ics = [_ic(nx, ny) for nx, ny in sizes]
    with Batch("heat", sizes, its=1, blocksize=16) as b:
        for i, (nx, _) in enumerate(sizes):
            b.set_constants(i, plugin_constants("heat", _globals(nx)))
            b.set_state(i, ics[i])
        for n in runs:
            b.run(n, graph=graph)
        got = [b.get_state(i) for i in range(len(sizes))]
    for u, ic in zip(got, ics):
        (ref,), _ = _solve(ic, _globals(ic.shape[1]), 1, 16, sum(runs), mode="standard", threads=256)
        assert np.array_equal(u, ref)
