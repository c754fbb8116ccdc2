"""The FP64 form where its integer arithmetic hands a particle back to the
FP64 instructions: positions on cell edges, next to them, at 0 and in the
first cells, mixed within warps with ordinary positions, with and without a
magnetic field.  Bit-exact against the oracle, as for ordinary particles."""
import numpy as np
import pytest

from cpic_gb300 import _lib
from tests import cases

pytestmark = pytest.mark.gpu


def edge_case(nx, ny, bz, L=2 * np.pi, seed=3):
    rng = np.random.default_rng(seed)
    Ly = L * ny / nx
    dx = L / nx

    def coords(n, side):
        k = rng.integers(0, side, n) * dx
        kinds = [k, k + 0.5 * dx, np.nextafter(k, np.inf), np.nextafter(k + dx, 0.0), k * 0.0,
                 np.full(n, 1e-300), np.full(n, 5e-324), k + dx * 2.0 ** -53, k + dx * 2.0 ** -30,
                 k + dx * rng.random(n)]
        v = np.choose(rng.integers(0, len(kinds), n), kinds)
        v = np.clip(v, 0.0, np.nextafter(side * dx, 0.0))
        # a position whose cell rounds to the one past the box is the
        # reference's out-of-range read (25 x 15 has some): not compared
        return np.where(np.floor(v * (1.0 / dx)) < side, v, 0.0)

    n = 4096
    x, y = coords(n, nx), coords(n, ny)
    ux, uy = (rng.choice([0.0, 0.1, -0.1, 2.0], n) * rng.choice([0.0, 1.0, 0.37], n) for _ in range(2))
    q = -L * Ly / n
    return dict(nx=nx, ny=ny, L=L, Ly=Ly, dt=0.05, B=(0.0, 0.0, bz), steps=3,
                species=[dict(q=q, m=-q, x=x, y=y, ux=ux, uy=uy)])


@pytest.mark.parametrize("nx,ny,bz", [(16, 16, 0.0), (16, 16, 0.7), (25, 15, 0.3), (64, 48, 0.0)])
def test_edge_positions_bitexact(lib, nx, ny, bz):
    case = edge_case(nx, ny, bz)
    g, o = cases.make_gpu(case, precision=_lib.FP64), cases.make_oracle(case)
    g.pre_step()
    o.pre_step()
    for it in range(3):
        ex, ey = o.E()
        g.set_E(ex, ey)
        o.stage_plasma_E()
        assert o.stage_plasma_r() == 0
        o.stage_field_rho()
        o.iter = o.iter + 1
        g.stage_plasma()
        for a, b in zip(g.particles(0), o.particles(0)):
            assert np.array_equal(a, b), it
        r_g, r_o = g.rho(), o.rho()
        assert np.max(np.abs(r_g - r_o)) <= 1e-12 * np.max(np.abs(r_o))
        o.stage_field_E()
    g.close()
