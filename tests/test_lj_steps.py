"""Steps of the mixed-precision LJ pass, whose kernel also makes the step's
update: every atom has to see its neighbours where they were before it.  Sizes
with eight, four and one thread per atom (the lines lie at 24,000 and 100,000
atoms), overflowed lists, and a batch, at 300 K.

A sequence of one step makes its update in kernels of their own, so ten steps
at once are compared with ten times one.  Both form the same FP32 forces from
the same FP32 positions; the half steps round differently in FP64 (1e-15 A), which
changes an FP32 position's rounding (1e-7 A) once in 1e9 and then an atom by
less than 1e-8 A.  A neighbour one step ahead (1e-3 A at 300 K) changes every
force by about 1e-4 Ha/A and every atom by 1e-6 A.  And two runs from one state
give the same bits."""
import numpy as np
import pytest

import comd_gb300 as cg
from comd_gb300.abi import by_id
from helpers import Case, world_by_id

pytestmark = pytest.mark.gpu


def lj(oracle, edges, seed=1):
    return Case(oracle, cg.POT_LJ, n=edges, bf=1.2, temp=300.0, amp=0.05, seed=seed)


def moved(c, x, y):
    box = np.array(list(c.s.contents.bounds))
    return np.abs(x - y - box * np.round((x - y) / box)).max()


@pytest.mark.parametrize("edges,cap", [((8, 7, 9), 0), ((19, 18, 20), 0), ((29, 30, 31), 0),
                                       ((8, 7, 9), 80)])
def test_steps(oracle, edges, cap):
    c = lj(oracle, edges)
    try:
        start = world_by_id(c.s)
        runs = [c.device(cg.PREC_MIXED) for _ in range(3)]
        out = []
        for d, n in zip(runs, (10, 10, 1)):
            assert d.list_info()[0]
            if cap:
                d.set_list_capacity(cap)
            for _ in range(10 // n):
                d.steps(n, 1e-15)
        for d in runs:
            d.download(c.s)
            d.close()
            out.append((world_by_id(c.s), by_id(c.s, "p")))
        assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
        assert moved(c, out[0][0], out[2][0]) < 1e-8
        assert moved(c, out[0][0], start) > 1e-2
    finally:
        c.close()


def test_batch(oracle):
    cases = [lj(oracle, (8, 7, 9)), lj(oracle, (7, 9, 8), seed=2)]
    try:
        runs = [cg.Batch([c.s for c in cases], cg.opts(cg.POT_LJ, cg.PREC_MIXED, True))
                for _ in range(2)]
        out = []
        for b, n in zip(runs, (10, 1)):
            assert b.list_info()[0]
            for _ in range(10 // n):
                b.steps(n, 1e-15)
        for b in runs:
            for r, c in enumerate(cases):
                b.download_rep(r, c.s)
                out.append(world_by_id(c.s))
            b.close()
        for r, c in enumerate(cases):
            assert moved(c, out[r], out[len(cases) + r]) < 1e-8
    finally:
        for c in cases:
            c.close()
