"""GPU test of the solute update where a diffusivity is zero or a concentration
vanishes: 1/GAMMA is infinite there, the harmonic mean and with it the flux are
zero, and the result is the concentration itself (conc_body.inc:62-133), not a
NaN.  The per-subroutine form and the fused steps against the C oracle."""
import numpy as np
import pytest

import make_golden as MG
import pyoracle as O
import pf3d
from conftest import RTOL_FP64, max_rel
from pf3d import deck

pytestmark = pytest.mark.gpu

# FP32: a relative rounding error of 2^-24 in c, phi and each of the ~20
# operations of a flux of at most c
TOL = {pf3d.PF_FP64: RTOL_FP64, pf3d.PF_FP32: 40 * 2.0 ** -24}


def setup(shape, **over):
    p = deck.run6_params(T0=922.0, taxa_resfr=19.84, AAA=0.01, **over)
    g = deck.grid(shape[0], shape[1], shape[2], 0.5e-6, 0.45e-6, 0.55e-6)
    st = MG.small_state(*shape, p)
    assert (st["phi"] > 0.95).any() and (st["phi"] < 0.05).any()
    return g, p, st


@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
@pytest.mark.parametrize("shape", [(33, 9, 17), (70, 41, 36)])
def test_no_diffusion_in_the_solid(gpu, shape, prec):
    g, p, st = setup(shape, D_sol=0.0)
    o = O.Oracle(g, p)
    o.load_state(st)
    o.concentracao_soluto()
    with pf3d.Domain(g, p, prec) as d:
        d.load_state(st)
        d.concentracao_soluto()
        assert max_rel(d.download("conc_soluto_new"), o.get(3)) <= TOL[prec]
        assert max_rel(d.download("conc_soluto_old"), o.get(2)) <= TOL[prec]


@pytest.mark.parametrize("fused", [0, 1])
@pytest.mark.parametrize("sweeps", [1, 2])
def test_no_diffusion_in_the_solid_steps(gpu, sweeps, fused):
    g, p, st = setup((70, 41, 36), D_sol=0.0, n_varreduras=sweeps)
    o = O.Oracle(g, p)
    o.load_state(st)
    o.step(3)
    want = o.fields()
    with pf3d.Domain(g, p) as d:
        d.set_option(pf3d.PF_OPT_FUSED, fused)
        d.load_state(st)
        d.step(3)
        got = d.fields()
    for k in want:
        assert max_rel(got[k], want[k]) <= RTOL_FP64, k


@pytest.mark.parametrize("small", [1e-160, 1e-250, 1e-300])
@pytest.mark.parametrize("fused,kernel", [(0, 1), (1, 1), (1, 0)])
def test_vanishing_concentration(gpu, fused, kernel, small):
    """A block of cells with next to no solute, inside the melt and across tiles:
    the reference gives finite values there, and so does every form."""
    g, p, st = setup((70, 41, 36))
    c = st["c"].copy()
    c[18:27, 10:30, 20:50] = small
    st = dict(st, c=c)
    o = O.Oracle(g, p)
    o.load_state(st)
    o.step(1)
    want = o.fields()
    assert np.isfinite(want["c"]).all()
    with pf3d.Domain(g, p) as d:
        d.set_option(pf3d.PF_OPT_FUSED, fused)
        d.set_option(pf3d.PF_OPT_KERNEL, kernel)
        d.load_state(st)
        d.step(1)
        got = d.fields()
    for k in want:
        assert max_rel(got[k], want[k]) <= RTOL_FP64, k
