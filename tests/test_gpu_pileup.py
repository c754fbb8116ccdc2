"""The mixed form's 32-bit weight sums at their limit: every particle exactly on
one node, so each adds the full 2^18 quanta to a single sum, for particle
counts around the overflow check's interval (31 chunks of 512 particles with 2
per thread, 62 of 256, 15 of 1024).  The charge on the node is exact."""
import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ppt", [1, 2, 4])
@pytest.mark.parametrize("n", [511, 512 * 31, 512 * 31 + 1, 512 * 62 + 7, 1024 * 47 + 3])
def test_every_particle_on_one_node(lib, n, ppt):
    ctx = _lib.Context(64, 64, 64.0, 64.0, 0.05, precision=_lib.MIXED, tile=8, halo=2, ppt=ppt)
    z = np.zeros(n)
    ctx.add_species(-1.0, 1.0, np.full(n, 10.0), np.full(n, 37.0), z, z)
    ctx.pre_step()
    rho = ctx.rho()
    ctx.close()
    want = np.zeros((64, 64))
    want[37, 10] = n
    assert np.array_equal(rho, want)
