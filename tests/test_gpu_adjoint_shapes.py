"""The adjoint run at the shapes where its particle order, blocks and deposit
regions change: grids smaller than a tile, one tile wide, larger tiles on sparse
grids, particle counts around a block's share, several sorts within the run,
particles at x = 0 and y = 0 (handed back to the FP64 instructions), with and
without a magnetic field; against the FP64 PyTorch re-implementation
differentiated by autograd."""
import math

import numpy as np
import pytest

from cpic_gb300 import _lib

pytestmark = pytest.mark.gpu

# FP64 rounding grows over the steps to about 1e-13 of the gradient's norm on
# the repository's adjoint workload; 1e-9 leaves room for the smallest plasmas
TOL = 1e-9


@pytest.mark.parametrize("nx,ny,n,steps,keep,bz", [
    (4, 4, 37, 12, 3, 0.0), (8, 64, 255, 20, 8, 0.4), (64, 8, 257, 20, 1, 0.0), (16, 16, 4096, 25, 9, 0.3),
    (256, 32, 1500, 18, 20, 0.0), (32, 32, 80001, 17, 4, 0.2), (512, 512, 3000, 6, 2, 0.0)])
def test_gradient_against_autograd(lib, nx, ny, n, steps, keep, bz):
    torch = pytest.importorskip("torch")
    from tests import adjoint_ref
    L = 2 * math.pi
    rng = np.random.default_rng(nx + 7 * ny + n)
    x, y = rng.random(n) * L, rng.random(n) * L
    x[:3], y[1:4] = 0.0, 0.0
    ux, uy = 0.3 * rng.standard_normal(n), 0.3 * rng.standard_normal(n)
    q = -L * L / n
    a = _lib.Adjoint(nx, ny, L, L, 0.05, 1.0, q, -q, n, steps, keep, Bz=bz, precision=_lib.FP64)
    for _ in range(2):                       # a second run on the same handle
        loss = a.forward(x, y, ux, uy)
        grads = a.backward()
    with pytest.raises(_lib.CpicError):      # refused, and the handle stays usable
        a.forward(np.full(n, L), y, ux, uy)
    a.close()
    t = [torch.from_numpy(v).clone().requires_grad_() for v in (x, y, ux, uy)]
    ref = adjoint_ref.field_energy(*t, nx, ny, L, 0.05, 1.0, q, -q, steps, Bz=bz)
    want = torch.autograd.grad(ref, t)
    assert abs(loss - float(ref)) <= TOL * abs(float(ref))
    for g, w in zip(grads, want):
        w = w.numpy()
        assert np.linalg.norm(g - w) <= TOL * np.linalg.norm(w)
