"""Several species in one launch of the fused kernel (layouts whose tiles leave
the GPU partly idle): identical to one launch per species, which 4 particles per
thread always takes, with two and three species, one of them empty, in both
forms."""
import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("nx,ny", [(64, 64), (50, 30)])
@pytest.mark.parametrize("counts", [(30000, 30000), (4000, 0, 90001), (7, 100000)])
def test_one_launch_for_all_species(lib, counts, nx, ny, precision):
    L = 2 * np.pi
    Ly = L * ny / nx
    rng = np.random.default_rng(len(counts) + nx)
    q = -L * Ly / max(counts)
    sp = []
    for k, n in enumerate(counts):
        sgn = 1.0 if k % 2 == 0 else -1.0
        sp.append((sgn * q, abs(q) * (1 + 50 * k), rng.random(n) * L, rng.random(n) * Ly,
                   0.3 * rng.standard_normal(n), 0.3 * rng.standard_normal(n)))
    out = []
    for ppt in (1, 2, 4):
        ctx = _lib.Context(nx, ny, L, Ly, 0.05, B=(0.0, 0.0, 0.4), precision=precision, ppt=ppt)
        for s in sp:
            ctx.add_species(*s)
        ctx.pre_step()
        ctx.run(10)
        out.append([ctx.rho(), *ctx.E()] + [a for k in range(len(sp)) for a in ctx.particles(k)])
        ctx.close()
    for other in out[:2]:
        for a, b in zip(other, out[2]):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("nx,ny,tile", [(256, 256, 8), (512, 256, 8), (150, 250, 0)])
def test_one_launch_over_several_waves(lib, nx, ny, tile, precision):
    """More tiles than the GPU holds blocks: 1024 (between one and two waves),
    2048 (over two), and a grid with ragged tiles; species of different density."""
    L = 2 * np.pi
    Ly = L * ny / nx
    rng = np.random.default_rng(nx + ny)
    counts = (400001, 90000, 250)
    q = -L * Ly / max(counts)
    sp = []
    for k, n in enumerate(counts):
        sgn = 1.0 if k % 2 == 0 else -1.0
        sp.append((sgn * q, abs(q) * (1 + 50 * k), rng.random(n) * L, rng.random(n) * Ly,
                   0.3 * rng.standard_normal(n), 0.3 * rng.standard_normal(n)))
    out = []
    for ppt in (1, 2, 4):
        ctx = _lib.Context(nx, ny, L, Ly, 0.02, B=(0.0, 0.0, 0.4), precision=precision, ppt=ppt,
                           tile=tile)
        for s in sp:
            ctx.add_species(*s)
        ctx.pre_step()
        ctx.run(10)
        out.append([ctx.rho(), *ctx.E()] + [a for k in range(len(sp)) for a in ctx.particles(k)])
        ctx.close()
    for other in out[:2]:
        for a, b in zip(other, out[2]):
            assert np.array_equal(a, b)
