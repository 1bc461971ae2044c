"""GPU test of the Karma passes' path for uniform neighbourhoods (phi exactly
+1 or -1 around a warp's row) against the C oracle, bit for bit: crystals and
melt with sharp walls anywhere against the tiles, single cells that break the
uniformity at a warp's edges, extents from one cell to ragged tiles, and a
non-finite U inside uniform regions (its NaNs must spread as in the oracle)."""
import numpy as np
import pytest

import pyoracle as O
from pf3d import karma

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 3), (31, 8, 2), (32, 9, 5), (33, 8, 6), (65, 17, 9), (40, 33, 140)]


def fields(nx, ny, nz, rng):
    phi = -np.ones((nz, ny, nx))
    phi[:, :, : nx // 2] = 1.0
    phi[nz // 2:, ny // 2:, :] = -1.0
    for _ in range(6):   # lone cells: 1 - ulp, a different sign, an interface value
        k, j, i = rng.integers(nz), rng.integers(ny), rng.integers(nx)
        phi[k, j, i] = rng.choice([np.nextafter(1.0, 0.0), -phi[k, j, i], 0.3, -np.nextafter(1.0, 0.0)])
    return phi, rng.uniform(-0.6, 0.0, phi.shape)


@pytest.mark.parametrize("Fn", [0.0, 0.02])
@pytest.mark.parametrize("shape", SHAPES)
def test_uniform_neighbourhoods_bit_identical(gpu, shape, Fn):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + 7 * ny + 31 * nz)
    p = karma.karma_params(nx=nx, ny=ny, nz=nz, Fnoise=Fn)
    phi, U = fields(nx, ny, nz, rng)
    for spoil in (None, np.inf, np.nan):
        u = U.copy()
        if spoil is not None:
            u[nz // 3, ny // 3, nx // 3] = spoil
        o = O.KarmaOracle(nx, ny, nz, p.lambda_, p.eps4, p.dx, p.dt, p.Fnoise, p.k)
        o.set(phi, u)
        with karma.Karma(p) as g:
            g.upload(phi, u)
            n = 4 if spoil is None else 1
            o.step(n)
            g.step(n)
            for name, a, b in zip(("phi", "U", "dphi"), g.fields(), o.get()):
                assert np.array_equal(a, b, equal_nan=True), (name, spoil)
