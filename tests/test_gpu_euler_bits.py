"""Euler level by level (csrc/euler_march.cuh) against the per-cell kernel
(Euler::step, threads=256) by bits, signs of zeros included: the factor 1/2 of a
cell's flux differences is folded into dt/dx only where it scales exactly, which
it does not where a difference is subnormal (momenta so small that their rows take
the plain divisions)."""
import numpy as np
import pytest

from test_gpu_euler_march import G, _field, _state

pytestmark = pytest.mark.gpu


def _subnormal(nx, ny, axis):
    """Uniform flow along one axis, momenta of 1 to 2^24 times the smallest
    subnormal across it: their flux differences are odd multiples of it, too."""
    rng = np.random.default_rng([nx, ny, axis])
    one = np.ones((nx, ny))
    q = _state(one, one if axis == 0 else 0 * one, one if axis == 1 else 0 * one, one)
    q[2 if axis == 0 else 1] = rng.integers(1, 1 << 24, (nx, ny)) * 2.0 ** -1074
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


@pytest.mark.parametrize("kind", ["vortex", "uniform", "steps", "below_two", "jumps", "subnormal0", "subnormal1"])
@pytest.mark.parametrize("nl", [1, 2, 7])
def test_march_has_the_per_cell_bits(kind, nl):
    ic = _subnormal(96, 128, int(kind[-1])) if kind[:-1] == "subnormal" else _field(kind, 96, 128)
    ref = _solve(ic, nl, "standard", threads=256)
    for mode in ("swept", "standard"):
        for a, b in zip(_solve(ic, nl, mode), ref):
            assert np.array_equal(_bits(a), _bits(b))
