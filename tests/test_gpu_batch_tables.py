"""A batch whose runs change block sizes: every run of another length brings a
table of (instance, block) units of its own, which the launches queued right after
it read.  Bitwise against the same fields advanced by single solvers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eq,its", [("heat", 1), ("euler", 2)])
@pytest.mark.parametrize("graph", [False, True])
def test_runs_of_many_lengths_in_a_row(eq, its, graph):
    from pysweep_b200 import Batch, Engine, plugin_constants
    from pysweep_b200.equations.euler import analytical_array
    sizes = [(32, 32), (256, 384), (64, 1056), (640, 96), (32, 64)]
    runs = (1, 5, 11, 2, 13, 4, 7, 3, 16, 9)
    rng = np.random.default_rng(8)
    ics, gs = [], []
    for i, (nx, ny) in enumerate(sizes):
        if eq == "heat":
            ics.append(rng.standard_normal((1, nx, ny)))
            gs.append([0.0, 1.0, 0.2 / nx / nx, 1 / nx, 1 / nx, 1.0, True])
        else:
            ics.append(analytical_array(nx, ny, 0.0, strength=2.0 + i))
            gs.append([0.0, 1.0, 0.01, 0.2, 0.2, 1.4])
    with Batch(eq, sizes, its=its, blocksize=16) as b:
        for i in range(len(sizes)):
            b.set_constants(i, plugin_constants(eq, gs[i]))
            b.set_state(i, ics[i])
        for n in runs:
            b.run(n, graph=graph)
        got = [b.get_state(i) for i in range(len(sizes))]
    for u, ic, g in zip(got, ics, gs):
        with Engine(eq, *ic.shape[1:], nv=ic.shape[0], its=its, blocksize=16) as e:
            for k, v in plugin_constants(eq, g).items():
                e.set_global(k, v)
            e.set_state(ic)
            e.run(sum(runs), mode="standard")
            assert np.array_equal(u, e.get_state())
