"""GPU test of the Karma passes' uniform path with parameters for which what is
left out there is not zero in the reference's expressions (a quotient 0/0 or a
product 0 times infinity): every field as the C oracle gives it."""
import numpy as np
import pytest

import pyoracle as O
from pf3d import karma

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [dict(eps4=1.0 / 3.0), dict(lambda_=np.inf), dict(Fnoise=np.inf), {}])
def test_uniform_cells_with_odd_parameters(gpu, over):
    nx, ny, nz = 40, 20, 24
    p = karma.karma_params(nx=nx, ny=ny, nz=nz, **over)
    phi = -np.ones((nz, ny, nx))
    phi[:, :, :12] = 1.0
    U = np.random.default_rng(5).uniform(-0.6, 0.0, phi.shape)
    o = O.KarmaOracle(nx, ny, nz, p.lambda_, p.eps4, p.dx, p.dt, p.Fnoise, p.k)
    o.set(phi, U)
    with karma.Karma(p) as g:
        g.upload(phi, U)
        o.step(1)
        g.step(1)
        for name, a, b in zip(("phi", "U", "dphi"), g.fields(), o.get()):
            assert np.array_equal(a, b, equal_nan=True), name
