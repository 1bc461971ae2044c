"""GPU test of objects created while the default stream is busy: their buffers
(the diagnostics' block counter among them) are cleared before anything is
uploaded or launched on their own streams, and not afterwards."""
import numpy as np
import pytest

import make_golden as MG
import pf3d
from pf3d import deck, karma

pytestmark = pytest.mark.gpu

SHAPE = (40, 24, 30)


def busy():
    """About 0.2 s of work queued on the default stream."""
    import torch
    a = torch.zeros(1 << 28, device="cuda")     # 1 GiB
    torch.cuda.synchronize()
    for _ in range(600):
        a.add_(1.0)
    done = torch.cuda.Event()
    done.record()
    return a, done


def setup():
    p = deck.run6_params(T0=922.0, taxa_resfr=19.84, AAA=0.01)
    return deck.grid(*SHAPE, 0.5e-6), p, MG.small_state(*SHAPE, p)


def run(g, p, st, done=None):
    with pf3d.Domain(g, p) as d, pf3d.Batch(pf3d.PF_FP64) as b:
        d.load_state(st)
        s = b.add(g, p)
        b.load_state(s, st)
        out = [b.diagnosticos(s), d.step_diag(2)]
        if done is not None:
            done.synchronize()
        b.step(2)
        d.step(2)
        return out + [b.diagnosticos(s), d.step_diag(1)], d.fields(), b.fields(s)


def test_domain_and_batch(gpu):
    case = setup()
    want = run(*case)
    hold, done = busy()
    got = run(*case, done)
    assert got[0] == want[0]
    for a, c in zip(got[1:], want[1:]):
        for k in c:
            assert np.array_equal(a[k], c[k]), k


def test_karma(gpu):
    nx, ny, nz = SHAPE
    p = karma.karma_params(nx=nx, ny=ny, nz=nz)
    rng = np.random.default_rng(2)
    phi, U = rng.uniform(-1, 1, (nz, ny, nx)), rng.uniform(-0.5, 0, (nz, ny, nx))
    hold, done = busy()
    with karma.Karma(p) as k:
        k.upload(phi, U)
        done.synchronize()
        assert np.array_equal(k.download(0), phi) and np.array_equal(k.download(1), U)
        k.step(1)
        k.sync()
