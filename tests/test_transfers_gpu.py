"""GPU test of the field transfers: what is uploaded comes back (rounded to
FP32 where the field is FP32), for pageable and pinned arrays, below, across
and above the staging chunks (one cell to several chunks a thread, rows longer
than a chunk), and from several threads at once."""
import threading

import numpy as np
import pytest

import pf3d
from pf3d import deck, karma

pytestmark = pytest.mark.gpu


def want(a, prec):
    return a if prec == 64 else a.astype(np.float32).astype(np.float64)


def values(shape, seed):
    a = np.random.default_rng(seed).normal(0, 1, shape)
    a.flat[0], a.flat[-1] = np.nan, np.inf
    return a


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("shape", [(5, 5, 5), (31, 40, 27), (64, 33, 16), (201, 130, 111), (37, 500, 640)])
def test_domain_and_batch_round_trip(gpu, shape, prec):
    import torch
    nx, ny, nz = shape
    g, p = deck.grid(nx, ny, nz, 0.5e-6), deck.run6_params()
    a = values((nz, ny, nx), nx)
    pinned = torch.from_numpy(a.copy()).pin_memory().numpy()
    with pf3d.Domain(g, p, prec) as d:
        for src in (a, pinned):
            d.upload("conc_soluto_old", src)
            out = torch.empty(nz, ny, nx, dtype=torch.float64).pin_memory().numpy()
            assert np.array_equal(d.download("conc_soluto_old"), want(a, prec), equal_nan=True)
            assert np.array_equal(d.download("conc_soluto_old", out), want(a, prec), equal_nan=True)
    with pf3d.Batch(prec) as b:
        s = b.add(g, p)
        b.upload(s, "TOLD", a)
        assert np.array_equal(b.download(s, "TOLD"), want(a, prec), equal_nan=True)
        b.upload(s, "TOLD", pinned)
        assert np.array_equal(b.download(s, "TOLD"), want(a, prec), equal_nan=True)


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("shape", [(1, 1, 1), (33, 7, 300), (1_100_000, 1, 2), (200, 200, 130)])
def test_karma_round_trip(gpu, shape, prec):
    nx, ny, nz = shape
    phi, U = values((nz, ny, nx), 1), values((nz, ny, nx), 2)
    with karma.Karma(karma.karma_params(nx=nx, ny=ny, nz=nz), prec) as k:
        k.upload(phi, U)
        assert np.array_equal(k.download(0), want(phi, prec), equal_nan=True)
        assert np.array_equal(k.download(1), want(U, prec), equal_nan=True)


def test_concurrent_threads(gpu):
    """Transfers of several objects from several threads, with steps queued
    on their streams, do not mix their fields."""
    shape, n = (70, 120, 140), 4
    bad = []

    def work(q):
        try:
            g, p = deck.grid(shape[2], shape[1], shape[0], 0.5e-6), deck.run6_params()
            with pf3d.Domain(g, p, 64 if q % 2 else 32) as d:
                a = np.random.default_rng(q).uniform(0.01, 0.02, shape)
                for r in range(4):
                    d.upload("conc_soluto_old", a + r)
                    d.upload("phase_field_old", np.zeros(shape))
                    d.upload("DPP", a * r)
                    if not np.array_equal(d.download("DPP"), want(a * r, 64 if q % 2 else 32)):
                        bad.append((q, r, "dpp"))
                    d.upload("conc_soluto_old", a)
                    d.step(3)
                    if not np.array_equal(d.download("phase_field_old"), np.zeros(shape)):
                        bad.append((q, r, "phi"))
        except Exception as e:   # reported by the main thread
            bad.append((q, repr(e)))

    ts = [threading.Thread(target=work, args=(q,)) for q in range(n)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
