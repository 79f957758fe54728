"""EAM tables that the packed forms (quartics per interval in FP64, records
staged in shared memory in mixed precision) do not take: phi and rho on
different grids, a start below zero, an end before the cutoff, more intervals than
either form holds, and one either side of the mixed form's 4,096.  Against the
oracle on the same tables, with the tolerances of the parity tests."""
import ctypes as C

import numpy as np
import pytest

import comd_gb300 as cg
from helpers import Case, compare_forces

interpolate = pytest.importorskip("scipy.interpolate")
pytestmark = pytest.mark.gpu


def resampled(t, x0, n):
    """the table's spline on n intervals from x0 to its end (constant below it)"""
    old = np.ctypeslib.as_array(t.values, (t.n + 1,)).copy()
    spline = interpolate.CubicSpline(t.x0 + np.arange(t.n + 1) / t.invDx, old)
    xn = t.x0 + t.n / t.invDx
    x = x0 + (np.arange(n + 3) - 1) * ((xn - x0) / n)
    v = np.ascontiguousarray(spline(np.clip(x, t.x0, xn)))
    t.x0, t.xn, t.invDx, t.n = x0, xn, n / (xn - x0), n
    t.values = C.cast(v.ctypes.data + 8, C.POINTER(C.c_double))
    return v


def shifted(t, d):
    t.x0 += d
    t.xn += d


def ended(t, xn):
    t.n = int((xn - t.x0) * t.invDx)
    t.xn = t.x0 + t.n / t.invDx


GRIDS = {
    "rho shifted": lambda p, r: shifted(r, 0.01),
    "rho coarser": lambda p, r: resampled(r, r.x0, r.n // 2),
    "below zero": lambda p, r: (resampled(p, -0.5, 3000), resampled(r, -0.5, 3000)),
    "ends early": lambda p, r: (ended(p, 4.5), ended(r, 4.5)),
    "4096": lambda p, r: (resampled(p, p.x0, 4096), resampled(r, r.x0, 4096)),
    "4097": lambda p, r: (resampled(p, p.x0, 4097), resampled(r, r.x0, 4097)),
    "80000": lambda p, r: (resampled(p, p.x0, 80000), resampled(r, r.x0, 80000)),
}


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("precision", [cg.PREC_FP64, cg.PREC_MIXED])
def test_table_grid(oracle, precision, grid):
    c = Case(oracle, cg.POT_EAM_TABLE, n=(7, 7, 8), temp=300.0)
    tables = [c.pot.ptr.contents.phi.contents, c.pot.ptr.contents.rho.contents]
    saved = [(t.n, t.x0, t.xn, t.invDx, C.cast(t.values, C.c_void_p).value) for t in tables]
    try:
        keep = GRIDS[grid](*tables)
        c.oracle_force()
        d = c.device(precision)
        e, _ = d.force()
        d.download(c.s)
        d.close()
        cmp = compare_forces(c.s, c.o)
        if precision == cg.PREC_FP64:
            assert cmp["f_max_rel"] < 1e-11 and cmp["e_max_rel"] < 1e-11, cmp
            assert cmp["rho_max_rel"] < 1e-12 and cmp["fi_max_rel"] < 1e-12, cmp
            assert abs(e - c.o.contents.e) <= 1e-12 * abs(c.o.contents.e)
        else:
            assert cmp["f_rel_rms"] < 1e-5 and cmp["f_max_rel"] < 1e-4, cmp
            assert cmp["rho_max_rel"] < 1e-6 and cmp["fi_max_rel"] < 1e-5, cmp
        del keep
    finally:
        for t, (n, x0, xn, inv, v) in zip(tables, saved):
            t.n, t.x0, t.xn, t.invDx = n, x0, xn, inv
            t.values = C.cast(v, C.POINTER(C.c_double))
        c.close()
