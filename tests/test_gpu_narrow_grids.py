"""Grids with a side of a few cells: the tile that the library chooses covers
that side and is below twice its length, and the run gives identical particles
and fields with it and with 4-cell tiles."""
import numpy as np
import pytest

from cpic_gb300 import _lib
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("nx,ny,n", [(4096, 8, 131072), (4096, 4, 262144), (4, 4096, 65536), (64, 4, 500),
                                     (2048, 16, 65536), (16, 16, 40), (8, 8, 100), (4, 4, 9)])
def test_chosen_tile_on_narrow_grids(lib, nx, ny, n, precision):
    cell = 2 * np.pi / nx / 0.05              # one cell per step
    case = cases.two_stream(nx=nx, ny=ny, n=n, v0=0.3 * cell, vth=0.05 * cell, Ly=2 * np.pi * ny / nx)
    out = []
    for tile in (0, 4):
        g = cases.make_gpu(case, precision=precision, tile=tile)
        T = g.tile_info()["tile_x"]
        assert T == 4 or T < 2 * min(nx, ny)
        g.pre_step()
        g.run(6)
        out.append((g.rho(), *g.E(), *g.particles(0)))
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
