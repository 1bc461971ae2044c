"""GPU test of a batch's defaults (the chunk that follows the membership, two
cells a thread in FP32) and of its trimmed step table: every field carries the
bits of the same batch with a fixed 64-plane chunk and one cell a thread,
while domains leave (a gap in the slots), join, stop at their target and the
membership goes from one tiny domain to many."""
import numpy as np
import pytest

import make_golden as MG
import pf3d
from pf3d import deck

pytestmark = pytest.mark.gpu


def case(nx, ny, nz, **over):
    p = deck.run6_params(T0=918.0, taxa_resfr=19.84, AAA=0.01, **over)
    return deck.grid(nx, ny, nz, 0.5e-6), p, MG.small_state(nx, ny, nz, p)


@pytest.mark.parametrize("over", [{}, dict(n_varreduras=1, ruido_tipo=2, h_quintico=1)])
@pytest.mark.parametrize("prec", [pf3d.PF_FP64, pf3d.PF_FP32])
def test_defaults_equal_fixed_shapes(gpu, prec, over):
    first = [case(5, 5, 5, **over), case(33, 9, 40, **over), case(40, 33, 131, **over)]
    later = [case(32, 32, 33, **over), case(70, 21, 64, **over)]

    def run(fixed):
        with pf3d.Batch(prec) as b:          # 4096 slots
            if fixed:
                b.set_tile(8, 64)
                b.set_paired(0)
            slots = []
            for g, p, st in first:
                slots.append(b.add(g, p))
                b.load_state(slots[-1], st)
            b.step(3)
            out = [b.fields(slots[0])]
            b.remove(slots[0])               # a gap below the slots in use
            b.set_target(slots[1], 9)
            b.step(9)
            b.remove(slots[2])
            for g, p, st in later:           # reuse both gaps
                s = b.add(g, p)
                b.load_state(s, st)
                slots.append(s)
            b.step(11)
            live = [slots[1], slots[3], slots[4]]
            out += [b.fields(s) for s in live]
            return out, [b.state(s).it for s in live]

    want, wit = run(True)
    got, git = run(False)
    assert git == wit == [9, 11, 11]
    for a, c in zip(got, want):
        for k in c:
            assert np.array_equal(a[k], c[k]), k
