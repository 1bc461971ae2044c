"""GPU test of the z-chunk rule: until PF_OPT_ZCHUNK is set the TMA passes take
the chunk that fills the GPU with the domain's tiles (one-plane chunks for the
smallest domains).  The chunk must not change a bit of any field, and the
option keeps reporting its documented default until it is set."""
import numpy as np
import pytest

import make_golden as MG
import pf3d
from pf3d import deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
@pytest.mark.parametrize("shape,over", [
    ((5, 5, 5), {}),                                  # one tile, fewer planes than a prologue
    ((33, 9, 48), {}),                                # two tiles: one-plane chunks
    ((64, 64, 65), dict(n_varreduras=1)),             # a last chunk shorter than the others
    ((40, 24, 130), dict(ruido_tipo=2, h_quintico=1)),
    ((97, 131, 40), dict(n_varreduras=3, ruido_tipo=1)),
])
def test_default_chunk_equals_fixed_chunks(gpu, prec, shape, over):
    p = deck.run6_params(T0=922.0, taxa_resfr=19.84, AAA=0.01, **over)
    g = deck.grid(*shape, 0.5e-6)
    st = MG.small_state(*shape, p)
    got = []
    for zc in (None, 64):
        with pf3d.Domain(g, p, prec) as d:
            if zc is not None:
                d.set_option(pf3d.PF_OPT_ZCHUNK, zc)
            v = pf3d._abi.C.c_int()
            pf3d._abi.LIB.pf_get_option(d.handle, pf3d.PF_OPT_ZCHUNK, pf3d._abi.C.byref(v))
            assert v.value == 64
            d.load_state(st)
            d.step(6)
            d.sync()
            got.append(d.fields())
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k]), k
