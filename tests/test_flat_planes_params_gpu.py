"""GPU test of uniform planes under parameters that make something else of the
zeros the passes leave out there (infinite or NaN factors), and with a
concentration at the pole of the driving force's logarithm: every field carries
the bits of the passes without that copy and of the cp.async passes."""
import numpy as np
import pytest

import pf3d
from pf3d import deck
from test_flat_planes_halo_gpu import check, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over,pole", [(dict(R=np.inf), None), (dict(AAA=np.inf), None), (dict(T0=np.nan), None),
                                       (dict(Ke=1.25), 1.0), (dict(Ke=1.25), 0.8)])
@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
def test_parameters_and_poles(gpu, prec, over, pole):
    kw = dict(T0=917.0, taxa_resfr=19.84, AAA=0.01)
    kw.update(over)
    st = state(160)
    if pole is not None:
        st["c"][350:360, 18, 40] = pole
    check(deck.run6_params(**kw), st, prec)
