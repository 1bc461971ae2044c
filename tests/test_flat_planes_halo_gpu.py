"""GPU test of where the passes that leave out uniform planes must not do so: a
non-finite or huge phase value two cells beside a uniform tile or two planes
below a uniform plane (the nodes next to it read it, and the zero differences
they are multiplied by do not absorb it).  Every field carries the bits of the
passes without that copy (short chunks) and of the cp.async passes."""
import numpy as np
import pytest

import pf3d
from pf3d import deck

pytestmark = pytest.mark.gpu

SHAPE = (97, 41, 452)


def state(melt_from):
    nx, ny, nz = SHAPE
    phi = np.zeros((nz, ny, nx))
    phi[:melt_from] = 1.0
    phi[melt_from:melt_from + 12] = (1 / (1 + np.exp(np.arange(-6, 6))))[:, None, None]
    c = 0.0196 * (1 - 0.86 * phi) * np.random.default_rng(3).uniform(0.99, 1.01, phi.shape)
    return {"phi": phi, "c": c, "T": np.full(phi.shape, 917.0), "dpp": np.full(phi.shape, 1e-5)}


def check(p, st, prec):
    g = deck.grid(*SHAPE, 0.5e-6)
    got = []
    for kernel, zc in ((1, 20), (1, 0), (1, 150), (0, 0)):
        with pf3d.Domain(g, p, prec) as d:
            d.set_option(pf3d.PF_OPT_KERNEL, kernel)
            d.set_option(pf3d.PF_OPT_ZCHUNK, zc)
            d.load_state(st)
            d.step(1)
            got.append(d.fields())
    for f in got[1:]:
        for k in f:
            assert np.array_equal(f[k], got[0][k], equal_nan=True), k


# cells in the second halo column or row of the tile of columns 32..63 and rows
# 16..23, one cell off its corner, and one of its own cells (two planes above
# it only the node between them sees it)
@pytest.mark.parametrize("x,y", [(30, 20), (65, 17), (45, 14), (40, 25), (31, 14), (50, 19)])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e30])
@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
def test_odd_value_two_cells_away(gpu, prec, value, x, y):
    st = state(160)                  # the first and the last 150-plane chunk are uniform
    st["phi"][390, y, x] = value     # in the melt
    st["phi"][70, y, x] = value      # in the crystal
    check(deck.run6_params(T0=917.0, taxa_resfr=19.84, AAA=0.01), st, prec)
