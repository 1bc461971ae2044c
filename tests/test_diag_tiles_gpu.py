"""GPU test of the diagnostics at the edges of its tiles, chunks and groups:
the five values against exactly rounded sums (1e-12, the plain form's bound) on
grids of one tile to several, with depths around the four-plane groups and the
chunk rule's limits, called twice (the kernel resets its own counter), and the
watchdog's count for non-finite cells placed on tile edges and walls."""
import math

import numpy as np
import pytest

import pf3d
from pf3d import deck
from pf3d._abi import PFError, PF_E_NONFINITE
from test_parity_gpu import exact_diagnostics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
@pytest.mark.parametrize("shape", [(5, 5, 5), (31, 7, 8), (32, 8, 9), (33, 9, 67), (64, 17, 64), (97, 41, 131),
                                   (200, 190, 66)])
def test_values_and_watchdog(gpu, shape, prec):
    nx, ny, nz = shape
    rng = np.random.default_rng(sum(shape))
    phi = rng.uniform(0, 1, (nz, ny, nx))
    c = rng.uniform(0.001, 0.08, phi.shape)
    if prec == pf3d.PF_FP32:
        phi, c = (v.astype(np.float32).astype(np.float64) for v in (phi, c))
    g = deck.grid(nx, ny, nz, 0.5e-6, 0.45e-6, 0.6e-6)
    with pf3d.Domain(g, deck.run6_params(), prec) as d:
        d.upload("phase_field_new", phi)
        d.upload("conc_soluto_new", c)
        dv = d.derived()
        ref = exact_diagnostics(phi, c, g.dx, g.dy, g.dz, dv.E0, dv.W0)
        for _ in range(2):
            for a, b in zip(d.diagnosticos(), ref):
                assert abs(a - b) <= 1e-12 * abs(b), (shape, a, b)
        spots = {(0, 0, 0), (nz - 1, ny - 1, nx - 1), (nz // 2, min(7, ny - 1), min(31, nx - 1)), (nz // 2, 0, nx - 1)}
        for name, bad in (("phase_field_new", np.nan), ("TNEW", np.inf)):
            f = phi.copy() if name == "phase_field_new" else np.full(phi.shape, 900.0)
            for q in spots:
                f[q] = bad
            d.upload(name, f)
            with pytest.raises(PFError) as e:
                d.diagnosticos()
            assert e.value.code == PF_E_NONFINITE and f": {len(spots)} cells" in str(e.value)
            if name == "phase_field_new":
                d.upload(name, phi)
        assert not math.isnan(ref[0])
