"""Euler level by level (csrc/euler_march.cuh) where its strips end and where its
quotients leave their safe ranges: grids narrower than a strip, one pair of
columns over it, single rows, odd level counts, runs that begin with either
stage, frames at any address; fields with vanishing and denormal momenta, uniform
regions (0/0 in the limiter), pressure jumps around the limiter's cut at 1e6,
densities a bit below a power of two, values beyond the safe ranges.  Every field
equals the per-cell kernel's (Euler::step, the plugin's operations in its order,
each rounded) bitwise, and the oracle's: the quotients are correctly rounded, so
the tolerance is zero."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

G = [0.0, 1.0, 0.01, 0.1, 0.1, 1.4]


def _state(rho, u, v, p):
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])


def _field(kind, nx, ny):
    rng = np.random.default_rng([nx, ny])
    one = np.ones((nx, ny))
    if kind == "vortex":
        from pysweep_b200.equations.euler import analytical_array
        return analytical_array(nx, ny, 0.0)
    if kind == "uniform":
        return _state(one, 0 * one, -0.0 * one, one)
    if kind == "steps":  # uniform blocks: no pressure step inside, none of momentum
        b = (np.add.outer(np.arange(nx) // 4, np.arange(ny) // 4) % 2).astype(float)
        return _state(1 + 7 * b, 0 * one, -0.0 * one, 1 + 7 * b)
    if kind == "below_two":  # densities whose mantissa is all ones, or nearly
        k = rng.integers(0, 4, (nx, ny))
        rho = (2 - k * 2.0 ** -52) * 2.0 ** rng.integers(-2, 3, (nx, ny))
        return _state(rho, rng.choice([0.0, 0.5, -0.25, 1e-17, 1e-300], (nx, ny)),
                      rng.standard_normal((nx, ny)), 1 + 1e-15 * rng.standard_normal((nx, ny)))
    if kind == "jumps":  # pressure steps of ratios around 1e6, and one ulp
        p = 1 + np.cumsum(rng.choice([0.0, 1e-6, 1e-12, 1.0, 2.0 ** -52], (nx, ny)), axis=1)
        return _state(1 + 0.1 * rng.random((nx, ny)), 0.3 * one, rng.choice([0.0, 1e-40], (nx, ny)), p)
    # extreme: a few cells beyond the safe ranges, or not physical at all
    q = _state(1 + rng.random((nx, ny)), rng.standard_normal((nx, ny)), 0 * one, one)
    for value in (1e30, 1e-200, -1.0, 5e-324, 1e120):
        q[rng.integers(0, 4), rng.integers(0, nx), rng.integers(0, ny)] = value
    return q


def _solve(ic, nl, bs, mode, gts0=1, frames=None, threads=0):
    from pysweep_b200 import Engine, plugin_constants
    _, nx, ny = ic.shape
    with Engine("euler", nx, ny, its=2, blocksize=bs) as e:
        for k, v in plugin_constants("euler", G).items():
            e.set_global(k, v)
        if threads:
            e.configure(threads=threads)
        e.set_state(ic)
        e.run(nl, mode=mode, gts0=gts0, frames=frames)
        e.synchronize()
        return e.get_state(0), e.get_state(1)


def _same(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("nx,ny,bs", [(8, 8, 8), (8, 56, 8), (16, 64, 8), (24, 120, 8), (40, 128, 8),
                                      (128, 32, 16), (640, 64, 32)])
@pytest.mark.parametrize("kind", ["vortex", "steps", "extreme"])
@pytest.mark.parametrize("nl,gts0", [(1, 1), (2, 1), (5, 2)])
def test_march_strips(nx, ny, bs, kind, nl, gts0):
    ic = _field(kind, nx, ny)
    ref = _solve(ic, nl, bs, "standard", gts0, threads=256)
    for mode in ("swept", "standard"):
        got = _solve(ic, nl, bs, mode, gts0)
        assert _same(got[0], ref[0]) and _same(got[1], ref[1])


@pytest.mark.parametrize("kind", ["vortex", "uniform", "steps", "below_two", "jumps", "extreme"])
def test_march_values(kind):
    ic = _field(kind, 96, 128)
    ref = _solve(ic, 6, 16, "standard", threads=256)
    got = _solve(ic, 6, 16, "swept")
    assert _same(got[0], ref[0]) and _same(got[1], ref[1])
    if kind in ("vortex", "steps", "below_two"):
        _, want, prev = oracle.standard("euler", ic, G, 2, 6, frames=False, euler_square="mul")
        assert _same(got[0], want) and _same(got[1], prev)


@pytest.mark.parametrize("off", [0, 1])
def test_march_frames_at_any_address(off):
    import torch
    nx, ny, nl = 32, 64, 6
    ic = _field("vortex", nx, ny)
    flat = torch.zeros(off + 3 * 4 * nx * ny, dtype=torch.float64, device="cuda")
    fr = flat[off:].view(3, 4, nx, ny)
    got = _solve(ic, nl, 16, "swept", frames=fr)
    want, _, _ = oracle.standard("euler", ic, G, 2, nl, euler_square="mul")
    assert _same(fr.cpu().numpy(), want[1:]) and _same(got[0], want[-1])


def test_batched_march_continues_and_mixes_stages():
    """Instances of many sizes in one launch; an odd run, then one instance set
    anew (its stages then alternate against the others'), then another run."""
    from pysweep_b200 import Batch, plugin_constants
    sizes = [(16, 16), (32, 64), (48, 128), (64, 16)]
    ics = [_field("vortex", *s) for s in sizes]
    with Batch("euler", sizes, its=2, blocksize=16) as b:
        for i in range(len(sizes)):
            b.set_constants(i, plugin_constants("euler", G))
            b.set_state(i, ics[i])
        b.run(5)
        b.set_state(1, ics[1])
        b.run(4)
        b.run(4)
        got = [(b.get_state(i, 0), b.get_state(i, 1)) for i in range(len(sizes))]
    for i, (a, older) in enumerate(got):
        ref = _solve(ics[i], 8 if i == 1 else 13, 16, "standard", threads=256)
        assert _same(a, ref[0]) and _same(older, ref[1])
