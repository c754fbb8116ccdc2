"""The library's own tile size need not divide the grid: the same plasma with
the chosen tiles (partly outside the grid in the last column and row) and with
tiles that divide it gives identical particles and fields, in both forms, at
particle counts on both sides of the rule's limits; a caller's tile still has
to divide."""
import numpy as np
import pytest

from cpic_gb300 import _lib
from tests import cases

pytestmark = pytest.mark.gpu


def runs(case, precision, tile, steps=8):
    g = cases.make_gpu(case, precision=precision, tile=tile)
    t = g.tile_info()["tile_x"]
    g.pre_step()
    g.run(steps)
    out = (g.rho(), *g.E(), *g.particles(0))
    g.close()
    return t, out


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("nx,ny,n,divides", [(50, 30, 1500, 2), (45, 75, 60000, 1), (98, 66, 400000, 2),
                                             (250, 150, 600011, 2), (36, 20, 100, 4), (333, 217, 30000, 1),
                                             (8, 6, 5000, 2), (5, 4, 300, 1)])
def test_chosen_tiles_change_nothing(lib, nx, ny, n, divides, precision):
    case = cases.two_stream(nx=nx, ny=ny, n=n, v0=0.4, vth=0.05, Ly=2 * np.pi * ny / nx)
    chosen, a = runs(case, precision, 0)
    _, b = runs(case, precision, divides)
    assert chosen in (4, 8, 16, 32)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_callers_tile_has_to_divide(lib):
    with pytest.raises(_lib.CpicError):
        _lib.Context(50, 30, 1.0, 0.6, 0.1, tile=4)
