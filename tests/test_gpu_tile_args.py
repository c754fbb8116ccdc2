"""cpic_create's tile arguments: one side given holds for both, stays when
particles are added, and has to be a power of two that divides the grid."""
import ctypes

import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu


def create(lib, nx, ny, tile_x, tile_y):
    p = _lib.Params()
    p.nx, p.ny, p.Lx, p.Ly, p.dt, p.e0 = nx, ny, float(nx), float(ny), 0.1, 1.0
    p.plasma_chunks, p.precision, p.tile_x, p.tile_y = 1, _lib.MIXED, tile_x, tile_y
    h = ctypes.c_void_p()
    return lib.cpic_create(ctypes.byref(p), ctypes.byref(h)), h


@pytest.mark.parametrize("tile_x,tile_y,want", [(0, 8, 8), (8, 0, 8), (0, 32, 32), (0, 16, 16), (4, 4, 4)])
def test_given_tile_stays(lib, tile_x, tile_y, want):
    r, h = create(lib, 64, 64, tile_x, tile_y)
    assert r == 0
    z = np.linspace(0.0, 63.9, 5000)
    d = z.ctypes.data_as(_lib.D)
    assert lib.cpic_add_species(h, -1.0, 1.0, len(z), d, d, d, d) == 0
    out = (ctypes.c_int32 * 4)()
    assert lib.cpic_tile_info(h, out) == 0
    lib.cpic_destroy(h)
    assert (out[0], out[1]) == (want, want)


@pytest.mark.parametrize("nx,ny,tile_x,tile_y", [(64, 64, 0, 24), (64, 64, 8, 16), (50, 30, 0, 32), (50, 30, 0, 4),
                                                 (64, 48, 0, 32), (50, 30, 4, 0)])
def test_refused_tiles(lib, nx, ny, tile_x, tile_y):
    r, _ = create(lib, nx, ny, tile_x, tile_y)
    assert r == -1
