"""GPU test of the passes that leave out what is zero on uniform planes (deep
domains in deep chunks): every field carries the bits of the same steps with
chunks too short for them, on states whose crystal and melt are exactly 1 and 0
over whole tiles, with walls anywhere against tiles and chunks, lone cells that
break the uniformity (an interface value, a last-bit difference, a negative
zero), concentrations outside the range in which the driving force's logarithm
is known to be finite, and a NaN."""
import numpy as np
import pytest

import pf3d
from pf3d import deck

pytestmark = pytest.mark.gpu


def state(nx, ny, nz, rng, spoil):
    phi = np.zeros((nz, ny, nx))
    phi[: nz // 3] = 1.0
    k0 = nz // 3
    phi[k0:k0 + 12] = (1 / (1 + np.exp(np.arange(-6, 6))))[:, None, None]
    phi[nz // 2:nz // 2 + 70, :, nx // 2:] = 1.0        # a wall across tiles
    for _ in range(25):
        k, j, i = rng.integers(3, nz - 3), rng.integers(ny), rng.integers(nx)
        phi[k, j, i] = rng.choice([0.3, np.nextafter(1.0, 0.0), 1e-300, -0.0, 1.0, 0.0])
    c = 0.0196 * (1 - 0.86 * phi) * rng.uniform(0.99, 1.01, phi.shape)
    if spoil:
        for v in (0.9, 0.14, 1e-12, np.nan):
            c[rng.integers(nz), rng.integers(ny), rng.integers(nx)] = v
    return {"phi": phi, "c": c, "T": np.full(phi.shape, 917.0), "dpp": rng.normal(0, 1e-4, phi.shape)}


@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
@pytest.mark.parametrize("shape,over", [((97, 41, 450), {}), ((130, 30, 520), dict(h_quintico=1, ruido_tipo=1))])
@pytest.mark.parametrize("spoil", [False, True])
def test_same_bits_as_short_chunks(gpu, shape, over, spoil, prec):
    p = deck.run6_params(T0=917.0, taxa_resfr=19.84, AAA=0.01, **over)
    g = deck.grid(*shape, 0.5e-6)
    st = state(*shape, np.random.default_rng(shape[0] + spoil), spoil)
    got = []
    for zc in (20, 64, 0, 450):
        with pf3d.Domain(g, p, prec) as d:
            d.set_option(pf3d.PF_OPT_ZCHUNK, zc)
            d.load_state(st)
            d.step(2 if spoil else 9)
            got.append(d.fields())
    for f in got[1:]:
        for k in f:
            assert np.array_equal(f[k], got[0][k], equal_nan=True), k
