"""The per-cell-courant solve and its adjoint in overlapped tiles
(csrc/heatvar_block.cuh) where tiles, launches and checkpoint segments end: grids
smaller than a tile, one over it, segments of one step, step counts that are no
multiple of a segment.  The forward field and lambda equal plain torch bitwise
(the same operations in the same order); dJ/dC, whose terms are fused
multiply-adds here, to the rounding of its sum: n terms, each off by at most half
an ulp of the running sum and one of the product, 2 n 2^-53 of the sum of their
magnitudes."""
import pytest

pytestmark = pytest.mark.gpu


def _lap(u, torch):
    return (((torch.roll(u, -1, 0) - 2 * u) + torch.roll(u, 1, 0)),
            ((torch.roll(u, -1, 1) - 2 * u) + torch.roll(u, 1, 1)))


def _plain(u, alpha, w, n, dt, dx, torch):
    h = torch.full_like(alpha, dx)  # (torch multiplies by the reciprocal of a scalar divisor)
    c = alpha * dt / h / h
    states = []
    for _ in range(n):
        states.append(u)
        xx, yy = _lap(u, torch)
        u = (c * xx + c * yy) + u
    lam, gc, size = w, torch.zeros_like(w), torch.zeros_like(w)
    for old in reversed(states):
        xx, yy = _lap(old, torch)
        gc, size = gc + lam * (xx + yy), size + (lam * (xx + yy)).abs()
        xx, yy = _lap(c * lam, torch)
        lam = lam + (xx + yy)
    f = dt / dx / dx
    return u, lam, gc * f, size * abs(f) * 2 * max(n, 1) * 2.0 ** -53


@pytest.mark.parametrize("nx,ny", [(3, 64), (17, 64), (48, 192), (49, 128), (200, 256), (1001, 448)])
@pytest.mark.parametrize("n,every", [(0, 4), (1, 1), (7, 3), (13, 64), (40, 16)])
def test_tiles_against_plain_torch(nx, ny, n, every):
    import torch
    from pysweep_b200.adjoint import heat_solve
    gen = torch.Generator(device="cuda").manual_seed(nx * 1000 + ny + n)
    rnd = lambda: torch.randn((nx, ny), dtype=torch.float64, device="cuda", generator=gen)  # noqa: E731
    u0, w = rnd(), rnd()
    alpha = 1 + 0.2 * torch.sin(rnd())
    dx = 1.0 / nx
    dt = 0.15 * dx * dx
    want, lam, galpha, tol = _plain(u0, alpha, w, n, dt, dx, torch)
    a, b = u0.clone().requires_grad_(), alpha.clone().requires_grad_()
    uT = heat_solve(a, b, n, dt, dx, every=every)
    g0, ga = torch.autograd.grad(uT, (a, b), w)
    assert torch.equal(uT, want) and torch.equal(g0, lam)
    assert ((ga - galpha).abs() <= tol).all()


@pytest.mark.parametrize("nx,ny,n,every", [(3, 64, 8, 8), (30, 64, 9, 9), (256, 320, 17, 17), (700, 768, 11, 6),
                                           (1600, 1536, 9, 9), (2100, 2112, 7, 7)])
def test_backward_tiles(nx, ny, n, every):
    """Levels backward in one launch, in tiles of every shape: grids smaller than
    a tile's halo, one over a tile, several tiles per SM."""
    test_tiles_against_plain_torch(nx, ny, n, every)


def test_recompute_stores_every_laplacian():
    import torch
    from pysweep_b200 import _lib
    from pysweep_b200.adjoint import _call, _p
    nx, ny, n = 90, 128, 21
    gen = torch.Generator(device="cuda").manual_seed(5)
    u = torch.randn((nx, ny), dtype=torch.float64, device="cuda", generator=gen)
    c = 0.1 + 0.05 * torch.rand((nx, ny), dtype=torch.float64, device="cuda", generator=gen)
    lap = torch.empty((n, nx, ny), dtype=torch.float64, device="cuda")
    work = torch.empty((2, nx, ny), dtype=torch.float64, device="cuda")
    _call(_lib.lib().ps_heatvar_recompute, _p(c), _p(u), _p(lap), n, nx, ny, _p(work))
    for k in range(n):
        xx, yy = _lap(u, torch)
        assert torch.equal(lap[k], xx + yy)
        u = (c * xx + c * yy) + u


def test_fields_at_odd_addresses():
    """Solver fields 8 bytes off a 16-byte boundary keep the shared-memory
    streams; the values are the same."""
    import torch
    from pysweep_b200 import Engine
    nx, ny, n = 64, 96, 9
    gen = torch.Generator(device="cuda").manual_seed(6)
    u = torch.randn((1, nx, ny), dtype=torch.float64, device="cuda", generator=gen)
    flat = torch.empty(nx * ny + 1, dtype=torch.float64, device="cuda")
    out = []
    for off in (0, 1):
        c = flat[off:off + nx * ny]
        c.copy_(0.1 + 0.01 * torch.arange(nx * ny, device="cuda") % 7 / 7)
        with Engine("heatvar", nx, ny, blocksize=32) as e:
            e.set_field(0, c)
            e.set_state(u)
            e.run(n)
            out.append(e.get_state())
    assert (out[0] == out[1]).all()
