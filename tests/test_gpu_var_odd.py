"""Per-cell-courant solvers whose fields lie 8 bytes off a 16-byte boundary run the
same overlapped tiles, two columns loaded one by one: one launch per several
levels, the values of aligned fields bitwise, Laplacians and sums included."""
import pytest

pytestmark = pytest.mark.gpu


def _run(eq, nx, ny, n, off, lap=None, frames=False):
    import torch
    from pysweep_b200 import Engine
    gen = torch.Generator(device="cuda").manual_seed(nx + ny)

    def field(k, values):
        f = torch.full((k * nx * ny + 1,), 7.0, dtype=torch.float64, device="cuda")
        f[off:off + k * nx * ny] = values.reshape(-1)
        return f, f[off:off + k * nx * ny]

    rnd = lambda k: torch.randn((k, nx, ny), dtype=torch.float64, device="cuda", generator=gen)  # noqa: E731
    u, c = rnd(2 if eq == "heatvar_adjoint" else 1), 0.1 + 0.01 * rnd(1)
    whole, parts = zip(*[field(1, c), field(n, rnd(n)), field(1, rnd(1))])
    with Engine(eq, nx, ny, blocksize=8) as e:
        e.set_field(0, parts[0])
        if lap or eq != "heatvar":
            e.set_field(1, parts[1])
            e.set_global("LEN", n)
        if eq == "heatvar_adjoint_mu":
            e.set_field(2, parts[2])
        e.set_state(u)
        e.profile(True)
        fr = torch.zeros((n // 3,) + tuple(u.shape), dtype=torch.float64, device="cuda") if frames else None
        e.run(n, frames=fr, frame_every=3)
        e.synchronize()
        kinds = {k: v[1] for k, v in e.profile_read().items() if v[1]}
        out = [torch.from_numpy(e.get_state()), parts[1].cpu(), parts[2].cpu()]
        out += [fr.cpu()] if frames else []
    # nothing beside the fields was written
    for f in whole:
        assert f[-1 if off == 0 else 0] == 7.0
    return out, kinds


@pytest.mark.parametrize("eq,lap", [("heatvar", False), ("heatvar", True), ("heatvar_adjoint_mu", False),
                                    ("heatvar_adjoint", False)])
@pytest.mark.parametrize("nx,ny,n", [(8, 8, 1), (16, 72, 7), (40, 64, 13), (64, 328, 16), (320, 600, 21)])
@pytest.mark.parametrize("frames", [False, True])
def test_odd_fields_take_the_tiles(eq, lap, nx, ny, n, frames):
    import torch
    if frames and n < 3:
        pytest.skip("no frame")
    want, _ = _run(eq, nx, ny, n, 0, lap, frames)
    got, kinds = _run(eq, nx, ny, n, 1, lap, frames)
    assert set(kinds) == {"block"} and (frames or kinds["block"] <= max(1, n // 3))
    for a, b in zip(got, want):
        assert torch.equal(a, b)
