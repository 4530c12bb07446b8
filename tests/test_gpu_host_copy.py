"""States read into host memory whose pages are mapped ahead of the copy: fresh
and used buffers, odd offsets, around the size from which pages are mapped (16 of
them).  The values arrive and no byte beside them changes."""
import ctypes
import mmap

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(32, 32), (64, 128), (96, 96), (256, 544)])
@pytest.mark.parametrize("offset", [0, 8, 4096, 12296])
def test_fresh_and_used_pages(nx, ny, offset):
    import numpy as np
    import torch
    from pysweep_b200 import Batch, Engine, _lib
    n = nx * ny * 8
    u = torch.rand((1, nx, ny), dtype=torch.float64, device="cuda")
    want = u.cpu().numpy().tobytes()
    buf = mmap.mmap(-1, offset + n + 8192)
    at = ctypes.addressof(ctypes.c_char.from_buffer(buf)) + offset
    with Engine("heat", nx, ny, blocksize=32) as e, Batch("heat", [(nx, ny)]) as b:
        e.set_state(u)
        b.set_state(0, u)
        for _ in range(2):  # fresh, then used
            _lib.check(_lib.lib().ps_get_state(e._h, ctypes.c_void_p(at), 0, 0), e._h)
            assert buf[offset:offset + n] == want
            assert not any(buf[:offset]) and not any(buf[offset + n:])
        fresh = np.empty((1, nx, ny))
        _lib.check(_lib.lib().ps_batch_get_state(b._h, 0, fresh.ctypes.data_as(ctypes.c_void_p), 0, 0),
                   b._h, batch=True)
        assert fresh.tobytes() == want
