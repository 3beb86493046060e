"""States fetched from a batch into pageable and into pinned arrays, at the edges of the fetch's chunks (4 MiB)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Euler cells of 32 bytes: below and at 1 MiB, one chunk and a row either way, two and three chunks, ragged
@pytest.mark.parametrize("nx,ny", [(128, 255), (128, 256), (512, 255), (512, 256), (512, 257), (512, 512), (512, 513), (700, 601)])
def test_fetch_into_pageable_and_pinned(hp, nx, ny):
    torch = pytest.importorskip("torch")
    c = hp.Config(system=hp.EULER, order=2, nx=nx, ny=ny, y_max=ny / nx, cfl=0.4, gamma1=1.4, pi1=0.0)
    U = hp.initial_state(c, "euler_quadrants", seed=nx + ny)
    with hp.Batch(max_instances=2, max_cells=nx * ny) as b:
        i = b.add(c, U, 0.0, 1e30, 0)
        assert b.get_state(i).tobytes() == U.tobytes()
        guarded = np.full(U.size + 16, 7.0)   # pageable, with a margin that has to stay
        pinned = torch.zeros(U.size, dtype=torch.float64).pin_memory().numpy()
        for out in (guarded[8:-8], pinned):
            st = hp.lib().hype_batch_get_state(b._h, i, out.ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
            assert st == hp.OK and out.tobytes() == U.tobytes()
        assert (guarded[:8] == 7.0).all() and (guarded[-8:] == 7.0).all()
