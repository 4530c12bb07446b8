"""ps_heatvar_forward with its output on its input: whatever the number of
launches, none writes the field it reads."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(48, 64), (200, 256), (640, 704)])
@pytest.mark.parametrize("n", [0, 1, 2, 4, 6, 8, 16, 18, 34, 35])
@pytest.mark.parametrize("every", [0, 4, 64])
def test_forward_in_place(nx, ny, n, every):
    import torch
    from pysweep_b200 import _lib
    from pysweep_b200.adjoint import _call, _p
    gen = torch.Generator(device="cuda").manual_seed(nx + n)
    u0 = torch.randn((nx, ny), dtype=torch.float64, device="cuda", generator=gen)
    alpha = 1 + 0.2 * torch.rand((nx, ny), dtype=torch.float64, device="cuda", generator=gen)
    out = []
    for inplace in (False, True):
        u = u0.clone()
        uT = u if inplace else torch.empty_like(u)
        ck = torch.zeros((max(1, -(-n // every)), nx, ny), dtype=u.dtype, device="cuda") if every else None
        courant, work = torch.empty_like(u), torch.empty_like(u)
        _call(_lib.lib().ps_heatvar_forward, _p(u), _p(alpha), _p(uT), nx, ny, n, 0.15 / nx / nx, 1.0 / nx,
              _p(courant), _p(work), _p(ck) if every else ctypes.c_void_p(), every or 64)
        torch.cuda.synchronize()
        out.append((uT, ck))
    assert torch.equal(out[0][0], out[1][0])
    assert not every or torch.equal(out[0][1], out[1][1])
