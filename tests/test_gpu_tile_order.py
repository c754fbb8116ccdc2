"""The fused kernel's tile order on uneven plasmas: whatever order the tiles
are taken in, every tile is taken exactly once, so a mixed run (exact integer
charge sums) gives bit-identical fields with a tile size whose tiles are
ordered each step (more tiles than blocks fit at once) and one whose tiles are
not.  Tile counts at and around the sort's ranges (1024 per round, 8192 at
most)."""
import numpy as np
import pytest

from cpic_gb300 import _lib
from tests import cases

pytestmark = pytest.mark.gpu


def uneven(nx, ny, n, seed):
    rng = np.random.default_rng(seed)
    L = 2 * np.pi
    Ly = L * ny / nx
    # half of the particles in a few clumps, half everywhere
    cx, cy = rng.random(5), rng.random(5)
    k = rng.integers(0, 5, n)
    clump = rng.random(n) < 0.5
    fx = np.where(clump, cx[k] + 0.02 * rng.standard_normal(n), rng.random(n)) % 1.0
    fy = np.where(clump, cy[k] + 0.02 * rng.standard_normal(n), rng.random(n)) % 1.0
    ux, uy = 0.2 * rng.standard_normal(n), 0.2 * rng.standard_normal(n)
    q = -L * Ly / n
    return dict(nx=nx, ny=ny, L=L, Ly=Ly, dt=0.05, B=(0.0, 0.0, 0.0), steps=12,
                species=[dict(q=q, m=-q, x=np.minimum(fx, 1 - 1e-12) * L, y=np.minimum(fy, 1 - 1e-12) * Ly,
                              ux=ux, uy=uy)])


@pytest.mark.parametrize("nx,ny,tile", [(128, 128, 4), (124, 132, 4), (256, 128, 4), (256, 256, 4),
                                        (360, 360, 4), (362, 362, 2)])
def test_order_takes_every_tile_once(lib, nx, ny, tile):
    case = uneven(nx, ny, 200000, nx + ny)
    big = 2 * tile if nx % (2 * tile) == 0 and ny % (2 * tile) == 0 else tile // 2
    out = []
    for t in (tile, big):
        g = cases.make_gpu(case, precision=_lib.MIXED, tile=t)
        g.pre_step()
        g.run(case["steps"])
        out.append((g.rho(), *g.E(), *g.particles(0)))
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
