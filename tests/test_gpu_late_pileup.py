"""The mixed form's 32-bit weight sums when a node fills up late: chunks of
particles on another node of the tile come first (left movers lead a tile's
particles after an upload), then as many on one node as would carry its sum past
2^32 units (16384 particles), around the overflow check's interval.  The charge
on both nodes is exact."""
import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ppt", [1, 2, 4])
@pytest.mark.parametrize("first,then", [(512 * 27, 512 * 34), (512 * 28 + 1, 512 * 33), (512 * 29 + 255, 20000),
                                        (512 * 30, 512 * 34), (1024 * 12, 16384), (1024 * 26 + 5, 40000)])
def test_node_that_fills_up_late(lib, first, then, ppt):
    n = first + then
    x, ux = np.full(n, 10.0), np.zeros(n)
    x[:first] = 13.0
    ux[:first] = -1e-9
    z = np.zeros(n)
    want = np.zeros((64, 64))
    want[37, 13], want[37, 10] = first, then
    for repeat in range(4):
        ctx = _lib.Context(64, 64, 64.0, 64.0, 0.05, precision=_lib.MIXED, tile=8, halo=2, ppt=ppt)
        ctx.add_species(-1.0, 1.0, x, np.full(n, 37.0), ux, z)
        ctx.pre_step()
        rho = ctx.rho()
        ctx.close()
        assert np.array_equal(rho, want)
