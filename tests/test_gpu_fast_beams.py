"""Plasmas that move several cells per step: many particles, or all, change tile
in every step.  No particle is lost, and the particle store has room for the
movers once it knows the plasma's speed."""
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


def kicked(grid, ppc, D, precision, **kw):
    """A plasma at rest whose first half step, under a given field, sets all of
    it to D cells per step without moving it."""
    x, y, _, z = beams(grid, ppc, D)
    c = _lib.Context(grid, grid, L, L, DT, precision=precision, **kw)
    c.add_species(-1e-12, 1e-12, x, y, z, z)
    c.pre_step()
    ex = np.full((grid + 1, grid), 2 * D * (L / grid) / DT / DT)
    c.set_E(ex, np.zeros_like(ex))
    c.stage_plasma()
    return c


@pytest.mark.parametrize("precision", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("D", [4.5, 5.5, 7.0])
def test_more_movers_than_the_arrivals_hold(lib, D, precision):
    """Most movers find their tile's arrivals full, and the spill list takes
    turns over all tiles until the next check, six steps on."""
    for repeat in range(3):
        c = kicked(64, 64, D, precision, tile=8)
        for k in range(3):
            c.run(6)
        assert c.status() == 0
        assert c.cell_counts().sum() == 64 * 64 * 64
        c.close()


def finishes(c, n, steps):
    for k in range(3):
        c.run(steps)
    last = c.layout_stats()["last_spill"]      # at the last check (a read-out counts anew)
    assert c.status() == 0
    assert c.cell_counts().sum() == n
    c.close()
    return last


HOT = [(64, 64, "beam", 2.5), (64, 64, "beam", 5.5), (64, 64, "beam", 12.0), (128, 16, "beam", 7.0),
       (256, 16, "beam", 8.0), (128, 128, "maxwellian", 5.5)]


@pytest.mark.parametrize("precision", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("tile", [0, 8])
@pytest.mark.parametrize("grid,ppc,kind,D", HOT)
def test_arrivals_hold_the_movers(lib, grid, ppc, kind, D, tile, precision):
    """Room for arrivals follows the speed of the plasma as it is loaded, in the
    library's tiles and in the caller's: nothing is lost, and next to nothing is
    spilled (an eighth of a per cent), in runs of eight steps between checks."""
    x, y, ux, uy = beams(grid, ppc, D)
    n = len(x)
    if kind == "maxwellian":               # D at 4.5 standard deviations
        rng = np.random.default_rng(6)
        s = D * (L / grid) / DT / 4.5
        ux, uy = s * rng.standard_normal(n), s * rng.standard_normal(n)
    c = _lib.Context(grid, grid, L, L, DT, precision=precision, tile=tile)
    c.add_species(-1e-12, 1e-12, x, y, ux, uy)
    c.pre_step()
    assert finishes(c, n, 8) < n / 800


@pytest.mark.parametrize("precision", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("grid,ppc,kind,D", HOT[:-1])
def test_faster_plasma_set_later(lib, grid, ppc, kind, D, precision):
    """The same for a plasma that is loaded at rest and then set to its speed."""
    x, y, ux, uy = beams(grid, ppc, D)
    n, z = len(x), np.zeros(len(x))
    c = _lib.Context(grid, grid, L, L, DT, precision=precision)
    c.add_species(-1e-12, 1e-12, x, y, z, z)
    c.set_particles(0, x, y, ux, uy)
    c.pre_step()
    assert finishes(c, n, 8) < n / 800


@pytest.mark.parametrize("precision", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("D", [2.5, 3.9])
def test_plasma_that_speeds_up(lib, D, precision):
    """A re-layout measures the speed again: a plasma at rest that a given field
    takes to D cells per step within 20 steps, each checked, then runs for eight
    steps between checks.  What is left in the spill list is less than a
    re-layout is made for (4096 records)."""
    x, y, _, z = beams(64, 64, D)
    n = len(x)
    c = _lib.Context(64, 64, L, L, DT, precision=precision)
    c.add_species(-1e-12, 1e-12, x, y, z, z)
    c.pre_step()
    ex = np.full((65, 64), -D * (L / 64) / DT / DT / 20)
    for k in range(21):
        c.set_E(ex, np.zeros_like(ex))
        c.stage_plasma()
    assert finishes(c, n, 8) <= 4096
