"""The library's tiles follow the largest species, in whatever order the species
are added: the tile is the one that species gets alone, and particles and fields
are those of 4-cell tiles.  A re-layout for a larger species carries the ones
already loaded over exactly."""
import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu
L = 2 * np.pi


def context(nx, ny, precision, tile, species, steps):
    c = _lib.Context(nx, ny, L, L * ny / nx, 0.02, B=(0.0, 0.0, 0.4), precision=precision, tile=tile)
    loaded = []
    for s in species:
        c.add_species(*s)
        loaded.append([a for k in range(len(loaded) + 1) for a in c.particles(k)])
    T = c.tile_info()["tile_x"]
    c.pre_step()
    c.run(steps)
    out = [c.rho(), *c.E()] + [a for k in range(len(species)) for a in c.particles(k)]
    c.close()
    return T, loaded, out


@pytest.mark.parametrize("precision", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("nx,ny", [(64, 64), (132, 60)])
@pytest.mark.parametrize("counts", [(0, 100000), (70, 100000), (100000, 0, 70), (70, 9000, 0, 262144)])
def test_tiles_follow_the_largest_species(lib, counts, nx, ny, precision):
    rng = np.random.default_rng(len(counts) + nx)
    q = -L * L * ny / nx / max(counts)
    species = [((-1) ** k * q, abs(q) * (1 + 50 * k), rng.random(n) * L, rng.random(n) * L * ny / nx,
                0.3 * rng.standard_normal(n), 0.3 * rng.standard_normal(n)) for k, n in enumerate(counts)]
    alone, _, _ = context(nx, ny, precision, 0, [species[int(np.argmax(counts))]], 0)
    T, loaded, out = context(nx, ny, precision, 0, species, 6)
    assert T == alone
    _, ref_loaded, ref = context(nx, ny, precision, 4, species, 6)
    for a, b in zip(out, ref):
        assert np.array_equal(a, b)
    for now, then in zip(loaded, ref_loaded):
        for a, b in zip(now, then):
            assert np.array_equal(a, b)
