"""GPU test of what gives the automatic z-chunk back.  64 planes is the value
the option and the batch report and start with, and it means the library's
choice: saving and restoring the option, or setting a batch's default tile,
must leave the passes as fast as one that was never touched (a fixed 64-plane
chunk is some ten times slower on the domain below), and an explicit chunk
changes no bit.  The autotuner must not end slower than the choice it starts
from, nor keep what it did not time."""
import numpy as np
import pytest

import make_golden as MG
import pf3d
from pf3d import deck
from pf3d._abi import C, LIB

pytestmark = pytest.mark.gpu

SHAPE = (36, 32, 48)
# the domain takes 19 us a step with its own chunk, 217 us with 64 planes:
# a factor of 3 stands far from both
SLACK = 3.0


def setup():
    p = deck.run6_params(T0=922.0, taxa_resfr=19.84, AAA=0.01)
    return deck.grid(*SHAPE, 0.5e-6), p, MG.small_state(*SHAPE, p)


def us_a_step(d, n=300):
    import torch
    d.step(20)
    d.sync()
    s = torch.cuda.Stream()
    d.set_stream(s.cuda_stream)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = 1e300
    for _ in range(3):
        e0.record(s)
        d.step(n)
        e1.record(s)
        e1.synchronize()
        best = min(best, 1e3 * e0.elapsed_time(e1) / n)
    d.set_stream(0)
    return best


def test_option_saved_and_restored(gpu):
    g, p, st = setup()
    with pf3d.Domain(g, p) as d:
        d.load_state(st)
        plain = us_a_step(d)
        v = C.c_int()
        LIB.pf_get_option(d.handle, pf3d.PF_OPT_ZCHUNK, C.byref(v))
        d.set_option(pf3d.PF_OPT_ZCHUNK, v.value)
        assert us_a_step(d) < SLACK * plain
        d.set_option(pf3d.PF_OPT_ZCHUNK, 48)
        d.step(1)
        d.set_option(pf3d.PF_OPT_ZCHUNK, v.value)
        assert us_a_step(d) < SLACK * plain


@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
@pytest.mark.parametrize("shape,over", [((33, 9, 48), {}), ((97, 131, 70), dict(n_varreduras=3, ruido_tipo=1)),
                                        ((64, 64, 130), dict(n_varreduras=1, ruido_tipo=2))])
def test_explicit_chunks_change_no_bit(gpu, shape, over, prec):
    p = deck.run6_params(T0=922.0, taxa_resfr=19.84, AAA=0.01, **over)
    g, st = deck.grid(*shape, 0.5e-6), MG.small_state(*shape, p)
    got = []
    for zc in (None, 63, 65):
        with pf3d.Domain(g, p, prec) as d, pf3d.Batch(prec) as b:
            if zc is not None:
                d.set_option(pf3d.PF_OPT_ZCHUNK, zc)
                b.set_tile(8, zc)
                b.set_paired(0)
            d.load_state(st)
            d.step(5)
            got.append(d.fields())
            if p.n_varreduras > 2:      # batches take one sweep or two
                continue
            s = b.add(g, p)
            b.load_state(s, st)
            b.step(5)
            got.append(b.fields(s))
    for f in got[1:]:
        for k in f:
            assert np.array_equal(f[k], got[0][k]), k


def batch_us(b, n=200):
    b.step(16)
    return min(1e3 * b.step(n) / n for _ in range(3))


def test_batch_tile_restored(gpu):
    g, p, st = setup()
    with pf3d.Batch(pf3d.PF_FP64) as b:
        b.load_state(b.add(g, p), st)
        plain = batch_us(b)
        b.set_tile(8, 40)
        b.step(1)
        b.set_tile(8, 64)
        assert batch_us(b) < SLACK * plain


def test_autotune_is_not_slower_and_keeps_only_what_it_timed(gpu):
    g, p, st = setup()
    with pf3d.Batch(pf3d.PF_FP64) as b:
        s = b.add(g, p)
        b.load_state(s, st)
        b.set_target(s, 1)
        b.step(1)                       # the slot has reached its target: nothing to time
        plain_it = b.state(s).it
        b.autotune(1)
        assert b.state(s).it == plain_it
        b.set_target(s, 0)
        untimed = batch_us(b)
    with pf3d.Batch(pf3d.PF_FP64) as b:
        s = b.add(g, p)
        b.load_state(s, st)
        plain = batch_us(b)
        assert untimed < SLACK * plain
        _, _, ms = b.autotune(20)
        assert ms > 0                   # timed here, not taken from the call that timed nothing
        assert batch_us(b) < 1.5 * plain
