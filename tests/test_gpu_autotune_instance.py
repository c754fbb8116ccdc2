"""cpic_autotune_tile times the kernel instance that a context with that tile
uses: the time it reports is the context's, to a tenth (timed with 2 particles
per thread, FP64 steps of this size take 1.23 times as long)."""
import math

import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu
L = 2 * math.pi


def test_reported_time_is_the_contexts(lib):
    n = 256 * 256 * 100
    T, ms = _lib.autotune_tile(256, 256, L, L, 0.05, n, 0.2, 0.0, precision=_lib.FP64)
    x, y, ux, uy = _lib.init_two_stream(1, 0, n, L, L, 0.2, 0.0, 0.01)
    c = _lib.Context(256, 256, L, L, 0.05, precision=_lib.FP64, tile=T)
    c.add_species(-L * L / n, L * L / n, x, y, ux, uy)
    c.pre_step()
    c.step()
    c.time_steps(3)
    own = min(c.time_steps(6)["ms_total"] / 6 for k in range(3))
    c.close()
    assert ms < 1.1 * own
