"""The FP64 rate epilogue's grid (CPU): within CUDA's limits for every window of the
meshes that a request may have (2^24 points), and every block of states and final
states taken once.  Two bands at every k of 81^3 or eight of 51^3 are more final
states than 65,535 blocks of them hold."""
import ctypes as ct

import numpy as np
import pytest

from elphbolt_gb300 import _lib, build


@pytest.fixture(scope="module")
def lib():
    build.build()
    L = _lib.load()
    L.ephg_debug_epilogue_grid.argtypes = [ct.c_int, ct.c_int, ct.POINTER(ct.c_int64)]
    L.ephg_debug_epilogue_grid.restype = ct.c_int
    return L


@pytest.mark.parametrize("nstates,nin", [(1, 1), (127, 16), (128, 17), (129, 1600), (1679, 1679), (300, 65535 * 16),
                                         (300, 65535 * 16 + 1), (8, 2 * 81**3), (40, 8 * 51**3), (1, 8 << 24)])
def test_grid_covers_all_blocks_within_the_limits(lib, nstates, nin):
    g = np.zeros(3, dtype=np.int64)
    assert lib.ephg_debug_epilogue_grid(nstates, nin, g.ctypes.data_as(ct.POINTER(ct.c_int64))) == _lib.EPHG_OK
    assert 0 < g[0] < 2**31 and 0 < g[1] <= 65535 and 0 < g[2] <= 65535
