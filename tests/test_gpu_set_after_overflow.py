"""cpic_set_particles on a species whose spill list holds records: they are
replaced with the rest, the count stays, and the state read back is the one set."""
import numpy as np
import pytest

from cpic_gb300 import _lib
from tests.test_gpu_ensemble_alone import CLUMP, REST, run_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("steps", [6, 7])
def test_spilled_records_are_replaced(lib, steps, prec):
    c, fresh = run_of(prec, 5), run_of(prec, 5)
    start = fresh.particles(0)
    c.run(steps)                   # the clump crosses and spills in move 5
    assert 0 < c.layout_stats()["last_spill"] < 4096
    c.set_particles(0, *start)
    assert c.cell_counts().sum() == CLUMP + REST
    for a, b in zip(c.particles(0), start):
        assert np.array_equal(a, b)
    c.step()
    assert c.cell_counts().sum() == CLUMP + REST and c.status() == 0
    c.close()
    fresh.close()
