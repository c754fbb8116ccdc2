"""The field solve at the sizes where its launch shapes change: one and two
columns per block (more or fewer than 304 spectrum columns), a last block
with a single column, radices 2, 3, 4, 5 and larger primes, an odd last row,
the smallest grid, against numpy's FP64 transform."""
import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu

# FP64: the bound used for phi elsewhere.  Mixed: the right-hand side and the
# spectrum are rounded to 24 bits (2^-24 each of the largest value) and about
# 2 log2(n) FP32 passes add as much again; 2e-6 is over 30 such roundings.
TOL = {_lib.FP64: 1e-12, _lib.MIXED: 2e-6}

SIZES = [(4, 4), (8, 4), (64, 64), (128, 32), (512, 256), (606, 16), (608, 16), (610, 24), (1216, 64),
         (1218, 20), (2048, 8), (16, 2048), (25, 15), (45, 75), (60, 100), (77, 13), (6, 10), (98, 9),
         (143, 121), (250, 150)]


def solve(rho):
    ny, nx = rho.shape
    c = 2.0 * (np.cos(2 * np.pi * np.arange(nx // 2 + 1) / nx)[None, :]
               + np.cos(2 * np.pi * np.arange(ny) / ny)[:, None]) - 4.0
    c[0, 0] = 1.0
    s = np.fft.rfft2(rho) / c
    s[0, 0] = 0.0
    return np.fft.irfft2(s, s=(ny, nx))


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_solve_shapes(lib, nx, ny, precision):
    rng = np.random.default_rng(nx * 1000 + ny)
    rho = rng.standard_normal((ny, nx))
    rho -= rho.mean()
    ctx = _lib.Context(nx, ny, float(nx), float(ny), 0.1, precision=precision)
    # one heavy and one opposite particle fix the fixed-point charge scale
    # and leave a neutral plasma (the mean that the mixed form removes is 0)
    ctx.add_species(1e3, 1.0, [0.5], [0.5], [0.0], [0.0])
    ctx.add_species(-1e3, 1.0, [0.5], [0.5], [0.0], [0.0])
    if precision == _lib.MIXED:
        # the mixed form's charge unit is the particle's / 2^18
        rho = np.round(rho * 2.0 ** 18 / 1e3) * (1e3 / 2.0 ** 18)
        rho -= np.round(rho.mean() * 2.0 ** 18 / 1e3) * (1e3 / 2.0 ** 18)
    ctx.set_rho(rho)
    ctx.stage_field_E()
    got, want = ctx.phi(), solve(rho)
    ctx.close()
    assert np.max(np.abs(got - want)) <= TOL[precision] * np.max(np.abs(want))
