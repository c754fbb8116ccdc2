"""Reading the mixed form's fields: the FP32 values widened exactly, on grids of
odd and of the smallest sides, without taking device memory."""
import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(4, 4), (5, 4), (4, 7), (6, 6), (33, 17), (250, 150), (64, 64), (241, 17), (64, 512)])
def test_fields_read_back_exactly(lib, nx, ny):
    rng = np.random.default_rng(nx + 1000 * ny)
    n = 40 * nx * ny
    c = _lib.Context(nx, ny, float(nx), float(ny), 0.05, precision=_lib.MIXED)
    z = np.zeros(n)
    c.add_species(-1.0 / 40, 1.0 / 40, rng.random(n) * nx, rng.random(n) * ny, z, z)
    c.pre_step()
    phi = c.phi()
    assert np.array_equal(phi, phi.astype(np.float32))
    # cells of unit width: E is half the difference of phi, exactly
    p = phi.astype(np.float32)
    ex, ey = c.E()
    want_x = (np.roll(p, 1, 1) - np.roll(p, -1, 1)) * np.float32(0.5)
    want_y = (np.roll(p, 1, 0) - np.roll(p, -1, 0)) * np.float32(0.5)
    for got, want in ((ex, want_x), (ey, want_y)):
        assert np.array_equal(got[:ny], want)
        assert np.array_equal(got[ny], got[0])
    wx = rng.standard_normal((ny + 1, nx)).astype(np.float32).astype(np.float64)
    wy = rng.standard_normal((ny + 1, nx)).astype(np.float32).astype(np.float64)
    wx[ny], wy[ny] = wx[0], wy[0]
    c.set_E(wx, wy)
    ex, ey = c.E()
    assert np.array_equal(ex, wx) and np.array_equal(ey, wy)
    c.close()


@pytest.mark.parametrize("nx,ny", [(64, 64), (72, 64), (130, 70)])
def test_reading_between_the_stages(lib, nx, ny):
    """Fields read after the field stage leave the particle stage as it is."""
    rng = np.random.default_rng(3)
    n = 20 * nx * ny
    x, y, u, v = rng.random(n) * nx, rng.random(n) * ny, rng.standard_normal(n), rng.standard_normal(n)
    out = []
    for read in (False, True):
        c = _lib.Context(nx, ny, float(nx), float(ny), 0.05, precision=_lib.MIXED)
        c.add_species(-1.0 / 20, 1.0 / 20, x, y, u, v)
        c.pre_step()
        for k in range(3):
            c.stage_field_E()
            if read:
                c.E()
                c.phi()
            c.stage_plasma()
        out.append((c.rho(), *c.E(), *c.particles(0)))
        c.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_reading_takes_no_device_memory(lib):
    torch = pytest.importorskip("torch")
    warm = _lib.Context(128, 128, 1.0, 1.0, 1e-3, precision=_lib.MIXED)     # (loads the kernels)
    warm.E()
    warm.phi()
    warm.close()
    c = _lib.Context(1024, 1024, 1.0, 1.0, 1e-3, precision=_lib.MIXED)
    c.add_species(-1.0, 1.0, [0.5], [0.5], [0.0], [0.0])
    c.pre_step()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    c.E()
    c.phi()
    assert torch.cuda.mem_get_info()[0] == before
    c.close()
