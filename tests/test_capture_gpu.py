"""GPU test of pf_step inside a stream capture: the passes are launched as
programmatic dependents of one another, and a captured block of steps, replayed
once, must give the bits of the same steps run directly; so must steps that
alternate with copies and diagnostics on the stream."""
import numpy as np
import pytest

import make_golden as MG
import pf3d
from pf3d import deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
@pytest.mark.parametrize("shape,over", [((36, 20, 24), {}), ((70, 45, 50), dict(n_varreduras=3, h_quintico=1))])
def test_captured_steps(gpu, shape, over, prec):
    import torch
    p = deck.run6_params(T0=922.0, taxa_resfr=19.84, AAA=0.01, **over)
    g = deck.grid(*shape, 0.5e-6)
    st = MG.small_state(*shape, p)
    with pf3d.Domain(g, p, prec) as a, pf3d.Domain(g, p, prec) as b:
        a.load_state(st)
        b.load_state(st)
        a.step(7)
        s = torch.cuda.Stream()
        b.set_stream(s.cuda_stream)
        b.step(1)          # every kernel is loaded before the capture
        b.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            b.step(4)
        graph.replay()
        torch.cuda.synchronize()
        for _ in range(2):
            b.step(1)
            b.step_diag(0)
            b.track()
        fa, fb = a.fields(), b.fields()
        for k in fa:
            assert np.array_equal(fa[k], fb[k]), k
        b.set_stream(None)
        del graph
