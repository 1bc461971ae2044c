"""GPU test of the per-subroutine passes (equacao_campo_fase and
concentracao_soluto as z-marching tiles with shared nodes).

With the gas constant zero the chemical driving force, the only part that
passes through `log`, drops out of the phase sweep, so DPP and the new phase
field must carry the oracle's bits: that pins every division of the reference
form (shared reciprocals with a correctly rounded last step) and the sharing
of nodes between cells, tiles and chunks.  The solute update keeps its
logarithms and is held to the plain form's 1e-12."""
import numpy as np
import pytest

import make_golden as MG
import pyoracle as O
import pf3d
from conftest import RTOL_FP64, max_rel
from pf3d import deck

pytestmark = pytest.mark.gpu

SHAPES = [(5, 5, 5), (32, 8, 6), (33, 9, 7), (64, 17, 70), (37, 29, 131), (97, 40, 12)]


def setup(shape, **over):
    p = deck.run6_params(T0=922.0, taxa_resfr=19.84, AAA=0.01, **over)
    g = deck.grid(shape[0], shape[1], shape[2], 0.5e-6, 0.45e-6, 0.55e-6)
    st = MG.small_state(*shape, p)
    rng = np.random.default_rng(sum(shape))
    st = dict(st, phi=np.clip(st["phi"] + rng.normal(0, 0.02, st["phi"].shape) * (st["phi"] > 1e-3), 0, 1))
    o = O.Oracle(g, p)
    o.load_state(st)
    return g, p, st, o


@pytest.mark.parametrize("over", [{}, dict(h_quintico=1, ruido_tipo=1), dict(ruido_tipo=2)])
@pytest.mark.parametrize("shape", SHAPES)
def test_phase_sweep_carries_the_oracles_bits(gpu, shape, over):
    g, p, st, o = setup(shape, R=0.0, **over)
    TP, M0 = o.scalars()["TP"], 1.9e-3
    with pf3d.Domain(g, p) as d:
        d.load_state(st)
        for it in (7, 8):
            o.set_scalars(it, TP, M0, 0.0)
            d.equacao_campo_fase(it, TP, M0)
            o.equacao_campo_fase()
            assert np.array_equal(d.download("DPP"), o.get(6))
            assert np.array_equal(d.download("phase_field_new"), o.get(1))
            d.copy_phase_new_to_old()
            o.set(0, o.get(1))


@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
@pytest.mark.parametrize("over", [{}, dict(h_quintico=1)])
@pytest.mark.parametrize("shape", SHAPES)
def test_solute_update(gpu, shape, over, prec):
    g, p, st, o = setup(shape, **over)
    with pf3d.Domain(g, p, prec) as d:
        d.load_state(st)
        d.concentracao_soluto()
        o.concentracao_soluto()
        # FP32: a relative rounding error of 2^-24 in c, phi and each of the
        # ~20 operations of a flux of at most c
        tol = RTOL_FP64 if prec == pf3d.PF_FP64 else 40 * 2.0 ** -24
        assert max_rel(d.download("conc_soluto_new"), o.get(3)) <= tol
        assert max_rel(d.download("conc_soluto_old"), o.get(2)) <= tol
