"""Plasmas loaded unevenly get smaller tiles than evenly spread ones of the same
count, the heavy tiles being what the particle kernel waits for; particles and
fields are those of any other tile, and a position in the box's last cell or an
empty species changes nothing."""
import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu
L = 2 * np.pi


def load(kind, nx, ny, n):
    rng = np.random.default_rng(nx + ny)
    x, y = rng.random(n), rng.random(n)
    if kind == "fifth":
        x, y = 0.3 + 0.2 * x, 0.2 + 0.2 * y
    elif kind == "bell":
        x, y = (0.5 + 0.1 * rng.standard_normal(n)) % 1.0, (0.5 + 0.1 * rng.standard_normal(n)) % 1.0
    elif kind == "corner":
        x, y = 1.0 - 0.02 * x, 1.0 - 0.02 * y
    hi = np.nextafter(1.0, 0.0)
    v = 0.1 * (L / nx) / 0.05
    return (np.minimum(x, hi) * L, np.minimum(y, hi) * L * ny / nx, v * rng.standard_normal(n),
            v * rng.standard_normal(n))


def run(nx, ny, precision, tile, particles):
    c = _lib.Context(nx, ny, L, L * ny / nx, 0.05, precision=precision, tile=tile)
    for p in particles:
        c.add_species(-1e-9, 1e-9, *p)
    T = c.tile_info()["tile_x"]
    c.pre_step()
    c.run(5)
    out = [c.rho(), *c.E()] + [a for k in range(len(particles)) for a in c.particles(k)]
    c.close()
    return T, out


@pytest.mark.parametrize("precision", [_lib.MIXED, _lib.FP64], ids=["mixed", "fp64"])
@pytest.mark.parametrize("kind,nx,ny,n,even", [("fifth", 256, 256, 500000, 8), ("bell", 512, 512, 1000000, 16),
                                               ("corner", 256, 256, 300000, 8), ("fifth", 250, 150, 300000, 8),
                                               ("fifth", 128, 16, 60000, None)])
def test_smaller_tiles_for_uneven_loads(lib, kind, nx, ny, n, even, precision):
    p = load(kind, nx, ny, n)
    T, out = run(nx, ny, precision, 0, [p])
    flat, _ = run(nx, ny, precision, 0, [load("even", nx, ny, n)])
    if even is not None:
        assert flat == even and T < even
    assert T <= flat
    given = 2 if nx % 4 or ny % 4 else 4 if T != 4 else 8
    _, ref = run(nx, ny, precision, given, [p])
    for a, b in zip(out, ref):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("order", [(0, 1, 2), (2, 1, 0), (1, 2, 0)])
def test_the_smallest_tile_of_the_large_species(lib, order):
    empty = [np.zeros(0)] * 4
    species = [load("even", 256, 256, 500000), load("fifth", 256, 256, 300000), empty]
    T, out = run(256, 256, _lib.MIXED, 0, [species[k] for k in order])
    assert T == 4
    _, ref = run(256, 256, _lib.MIXED, 16, [species[k] for k in order])
    for a, b in zip(out, ref):
        assert np.array_equal(a, b)
