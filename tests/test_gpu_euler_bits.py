"""Euler level by level (csrc/euler_march.cuh) against the per-cell kernel
(Euler::step, threads=256) by bits, signs of zeros included: the factor 1/2 of a
cell's flux differences is folded into dt/dx only where it scales exactly, which
it does not where a difference is subnormal (momenta so small that their rows take
the plain divisions)."""
import numpy as np
import pytest

from test_gpu_euler_march import G, _field, _state

pytestmark = pytest.mark.gpu


def _subnormal(nx, ny, kind):
    """Uniform flow along one axis, momenta of multiples of the smallest subnormal
    across it, so that their flux differences are odd multiples of it, too: 1 to
    2^24 of them, a few of either sign and zeros of both, or those in a few rows
    and columns only."""
    rng = np.random.default_rng([nx, ny, len(kind)])
    one, axis = np.ones((nx, ny)), int(kind[-1])
    q = _state(one, one if axis == 0 else 0 * one, one if axis == 1 else 0 * one, one)
    many = rng.integers(1, 1 << 24, (nx, ny)) * 2.0 ** -1074
    few = rng.choice([-3.0, -2.0, -1.0, -0.0, 0.0, 1.0, 2.0, 3.0], (nx, ny)) * 2.0 ** -1074
    if kind.startswith("many"):
        v = many
    elif kind.startswith("few"):
        v = few
    else:
        v = np.full((nx, ny), -0.0)
        for at in ((10, slice(None)), (11, slice(30, 34)), (57, slice(0, 3)), (slice(40, 44), 70)):
            v[at] = few[at]
    q[2 if axis == 0 else 1] = v
    return q


def _solve(ic, nl, mode, threads=0, consts=()):
    from pysweep_b200 import Engine, plugin_constants
    _, nx, ny = ic.shape
    with Engine("euler", nx, ny, its=2, blocksize=16) as e:
        for k, v in {**plugin_constants("euler", G), **dict(consts)}.items():
            e.set_global(k, v)
        if threads:
            e.configure(threads=threads)
        e.set_state(ic)
        e.run(nl, mode=mode)
        return e.get_state(0), e.get_state(1)


def _bits(a):
    return np.ascontiguousarray(a).view(np.int64)


@pytest.mark.parametrize("kind", ["vortex", "uniform", "steps", "below_two", "jumps", "many0", "many1", "few0", "few1",
                                  "some0", "some1"])
@pytest.mark.parametrize("nl", [1, 2, 7])
def test_march_has_the_per_cell_bits(kind, nl):
    ic = _subnormal(96, 128, kind) if kind[-1] in "01" else _field(kind, 96, 128)
    ref = _solve(ic, nl, "standard", threads=256)
    for mode in ("swept", "standard"):
        for a, b in zip(_solve(ic, nl, mode), ref):
            assert np.array_equal(_bits(a), _bits(b))
