"""Every tile of the overlapped blocks, and the streams, on the smallest grids that
are planned to take them (test_host_block_shapes.py checks that they do), bitwise:
heat against the per-cell kernel or the float32 oracle, alone and as a batch of one;
the per-cell-courant forms against the shared-memory prisms; the backward tiles
against plain torch."""
import numpy as np
import pytest

import oracle
from block_grids import GRIDS
from test_gpu_block import _globals, _ic, _solve
from test_gpu_var_block import test_tiles_against_plain_torch as against_plain_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nl", GRIDS["fe"])
def test_forward_euler(nx, ny, nl):
    from pysweep_b200 import Batch, plugin_constants
    ic, g = _ic(nx, ny), _globals(nx)
    (got,), _ = _solve(ic, g, 1, 32, nl)
    (ref,), _ = _solve(ic, g, 1, 32, nl, mode="standard", threads=256)
    assert np.array_equal(got, ref)
    with Batch("heat", [(nx, ny)], blocksize=32) as b:
        b.set_constants(0, plugin_constants("heat", g))
        b.set_state(0, ic)
        b.run(nl)
        assert np.array_equal(b.get_state(0), ref)


@pytest.mark.parametrize("nx,ny,nl", GRIDS["f32"])
def test_float32(nx, ny, nl):
    ic, g = _ic(nx, ny).astype(np.float32), _globals(nx)
    (got,), _ = _solve(ic, g, 1, 32, nl, dtype="float32")
    assert np.array_equal(got, oracle.heat_f32(ic, g, nl))


@pytest.mark.parametrize("nx,ny,nl", GRIDS["rk2"])
def test_two_stages(nx, ny, nl):
    ic, g = _ic(nx, ny), _globals(nx, False)
    got, _ = _solve(ic, g, 2, 32, nl)
    ref, _ = _solve(ic, g, 2, 32, nl, mode="standard", threads=256)
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))


def _var(eq, nx, ny, nl, lap, threads):
    import torch
    from pysweep_b200 import Engine
    gen = torch.Generator(device="cuda").manual_seed(nx + ny)
    rnd = lambda k: torch.randn((k, nx, ny), dtype=torch.float64, device="cuda", generator=gen)  # noqa: E731
    u, c, laps, acc = rnd(2 if eq == "heatvar_adjoint" else 1), 0.1 + 0.01 * rnd(1), rnd(nl), rnd(1)
    with Engine(eq, nx, ny, blocksize=32) as e:
        e.configure(threads=threads)
        e.set_field(0, c)
        if lap:
            e.set_field(1, laps)
            e.set_global("LEN", nl)
        if eq == "heatvar_adjoint_mu":
            e.set_field(2, acc)
        e.set_state(u)
        e.run(nl)
        return torch.from_numpy(e.get_state()), laps.cpu(), acc.cpu()


@pytest.mark.parametrize("eq,nx,ny,nl", [
    *(("heatvar", *g) for g in GRIDS["forward"]), *(("recompute", *g) for g in GRIDS["recompute"]),
    *((eq, *g) for eq in ("heatvar_adjoint_mu", "heatvar_adjoint") for g in GRIDS["adjoint"])])
def test_courant_number_per_cell(eq, nx, ny, nl):
    import torch
    lap, eq = eq != "heatvar", "heatvar" if eq == "recompute" else eq
    for a, b in zip(_var(eq, nx, ny, nl, lap, 128), _var(eq, nx, ny, nl, lap, 256)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("nx,ny,nl", GRIDS["backward"])
def test_backward(nx, ny, nl):
    against_plain_torch(nx, ny, nl, nl)
