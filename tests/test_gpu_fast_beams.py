"""Plasmas that move several cells per step: many particles change tile in
every step, and no particle is lost."""
import math

import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu
L = 2 * math.pi
DT = 0.05


def beams(grid, ppc, D, seed=5):
    """Two beams of D cells per step in opposite directions."""
    n = grid * grid * ppc
    rng = np.random.default_rng(seed)
    x, y = rng.random(n) * L, rng.random(n) * L
    v = D * (L / grid) / DT
    return x, y, np.where(rng.random(n) < 0.5, v, -v), np.zeros(n)


@pytest.mark.parametrize("precision", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("D", [4.5, 5.5, 7.0])
def test_more_movers_than_the_arrivals_hold(lib, D, precision):
    """A plasma loaded at rest and then set to beams: most movers find their
    tile's arrivals full and the spill list takes turns over all tiles until
    the next check, six steps on."""
    x, y, ux, uy = beams(64, 64, D)
    n, z = len(x), np.zeros(len(x))
    for repeat in range(3):
        c = _lib.Context(64, 64, L, L, DT, precision=precision, tile=8)
        c.add_species(-L * L / n, L * L / n, x, y, z, z)
        c.set_particles(0, x, y, ux, uy)
        c.pre_step()
        for k in range(3):
            c.run(6)
        assert c.status() == 0
        assert c.cell_counts().sum() == n
        c.close()
