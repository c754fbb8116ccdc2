"""A run stepped alternately by its own calls and by an ensemble's graph gives
what the same run stepped alone gives: a clump of particles that crosses into
the next tile, and overflows its arrivals, during a replay of the graph is still
there after the run's next own step; charge is deposited on a cleared grid when
a field stage was issued before the replay."""
import math

import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu
L = 2 * math.pi
DT = 0.05
CLUMP, REST = 2000, 20000


def run_of(prec, lead):
    """64 x 64 cells in 8-cell tiles: REST particles at rest, and a clump that
    moves one cell per step, reaches the next tile's edge in move `lead` and then
    spills about 1800 records (a rebuild starts at 4096)."""
    cell = L / 64
    rng = np.random.default_rng(11)
    x = np.concatenate([rng.random(REST) * L, (24 - lead + 0.3 + 0.4 * rng.random(CLUMP)) * cell])
    y = np.concatenate([rng.random(REST) * L, (20 + 4 * rng.random(CLUMP)) * cell])
    ux = np.concatenate([np.zeros(REST), np.full(CLUMP, cell / DT)])
    c = _lib.Context(64, 64, L, L, DT, 1.0, precision=prec, tile=8, halo=1)
    c.add_species(-1e-30, 1e-30, x, y, ux, np.zeros_like(ux))
    c.pre_step()
    return c


def same(c, ref):
    assert c.iter == ref.iter
    assert c.status() == 0
    assert c.cell_counts().sum() == CLUMP + REST
    assert np.array_equal(c.rho(), ref.rho())
    for a, b in zip(c.particles(0), ref.particles(0)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("lead", [5, 6])
@pytest.mark.parametrize("odd", [False, True], ids=["own step", "odd step"])
def test_records_spilled_by_a_replay(lib, odd, lead, prec):
    c, ref = run_of(prec, lead), run_of(prec, lead)
    ens = _lib.Ensemble([c])
    ens.run(3)                     # iteration 0 and one pair: captured
    c.run(2)                       # own steps: the lists are read as empty
    assert c.layout_stats()["last_spill"] == 0
    if odd:
        ens.run(3)                 # a pair replayed, then an eager step
    else:
        ens.run(2)
        c.step()
    ref.run(8)
    same(c, ref)
    c.run(3)
    ref.run(3)
    same(c, ref)
    ens.close()


@pytest.mark.parametrize("prec", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
def test_field_stage_before_a_replay(lib, prec):
    c, ref = run_of(prec, 20), run_of(prec, 20)
    ens = _lib.Ensemble([c])
    ens.run(3)
    c.stage_field_E()
    ens.run(2)
    c.stage_plasma()
    ref.run(5)
    ref.stage_plasma()
    same(c, ref)
    ens.close()
