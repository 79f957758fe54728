"""comdgb_sim_set_cheby with intervals that need longer FP64 tables than the ones
before (the pair series from 1 A and the density to 4 times its end), shorter
ones, and the first again: the tables are made anew each time, so every step
gives the bits of a handle that has seen nothing else."""
import numpy as np
import pytest

import comd_gb300 as cg
from comd_gb300.abi import by_id
from helpers import Case
from test_adjoint import cheb_base

pytestmark = pytest.mark.gpu


def test_tables_grow_and_shrink(oracle):
    c = Case(oracle, cg.POT_EAM_CHEBY, n=(6, 6, 7), temp=300.0)
    try:
        coef, x0, xn = cheb_base(c)
        wide0, wide1 = x0.copy(), xn.copy()
        wide0[:2] = 1.0
        wide1[2] *= 4.0
        narrow0 = x0.copy()
        narrow0[:2] = 2.4
        sets = [(x0, xn), (wide0, wide1), (narrow0, xn), (x0, wide1), (x0, xn)]

        def forces(d, which):
            d.set_cheby(coef, *sets[which])
            e, _ = d.force()
            d.download(c.s)
            return e, by_id(c.s, "f")

        d = c.device(cg.PREC_FP64)
        for which in range(len(sets)):
            e, f = forces(d, which)
            alone = c.device(cg.PREC_FP64)
            e1, f1 = forces(alone, which)
            alone.close()
            assert e == e1 and np.array_equal(f, f1), which
        d.close()
    finally:
        c.close()
