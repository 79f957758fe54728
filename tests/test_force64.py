"""The FP64 passes against the oracle where their shape changes: either side of
12,000 atoms (16 and 4 threads an atom) and past 2^19 (one), with an atom taken
out so that the atoms do not fill the last warp, and box widths that put the
fixed-point unit on both sides of a power of two (LJ cutoffs of 3.9 and 4.1 A).
A table's intervals are polynomials in r^2 up to the cutoff, the ones near its
lower end the formula: pairs are put on both sides of every end there, and below
the table.  Tolerances as in the FP64 parity tests: the sums differ in order alone."""
import pytest

import comd_gb300 as cg
from comd_gb300.abi import slot_views
from helpers import Case, compare_forces
from test_fo_lanes import without_last_atom

pytestmark = pytest.mark.gpu


def check(c):
    c.oracle_force()
    d = c.device(cg.PREC_FP64)
    e, _ = d.force()
    d.download(c.s)
    d.close()
    cmp = compare_forces(c.s, c.o)
    assert cmp["f_max_rel"] < 1e-11 and cmp["e_max_rel"] < 1e-11, cmp
    if c.potential != cg.POT_LJ:
        assert cmp["rho_max_rel"] < 1e-12 and cmp["fi_max_rel"] < 1e-12, cmp
    assert abs(e - c.o.contents.e) <= 1e-12 * abs(c.o.contents.e)


@pytest.mark.parametrize("potential", [cg.POT_EAM_TABLE, cg.POT_EAM_CHEBY, cg.POT_LJ])
@pytest.mark.parametrize("edges", [(7, 6, 8), (15, 14, 15)])
def test_threads_per_atom(oracle, potential, edges):
    c = Case(oracle, potential, n=edges, temp=300.0)
    try:
        without_last_atom(c)
        check(c)
    finally:
        c.close()


def test_one_thread_per_atom(oracle):
    c = Case(oracle, cg.POT_EAM_TABLE, n=(51, 51, 51), temp=300.0)
    try:
        without_last_atom(c)
        check(c)
    finally:
        c.close()


@pytest.mark.parametrize("cutoff", [3.9, 4.1])
def test_fixed_point_unit(oracle, cutoff):
    c = Case(oracle, cg.POT_LJ, n=(7, 7, 8), temp=300.0, amp=0.03)
    pot = cg.lj_potential(2.315, 0.167 / 27.211386245988, cutoff, 63.55)
    try:
        oracle.free(c.o)
        cg.free_host(c.s)
        c.pot, c.s = pot, cg.fcc(7, 7, 8, 3.615, 1.0, 1.0, pot)
        cg.seed(c.s, 3, cg.DISP_GAUSSIAN, 0.03, 300.0, 63.55)
        assert oracle.rebox(c.s) == 0
        c.o = oracle.clone(c.s)
        check(c)
    finally:
        c.close()


# distances in table intervals from the table's lower end; the derivative jumps
# at 1 and 0 (its first interval counts as flat), so none lies on an end
@pytest.mark.parametrize("at", [-200.3, -0.5, 0.5, 0.9999, 1.0001, 1.5, 1.9999, 2.0001, 7.3, 150.2])
def test_close_pair_of_a_table(oracle, at):
    c = Case(oracle, cg.POT_EAM_TABLE, n=(6, 6, 7), temp=300.0, amp=0.03)
    try:
        phi = c.pot.ptr.contents.phi.contents
        v = slot_views(c.s)
        assert v["natoms"][0] > 1
        v["r"][1] = v["r"][0]
        v["r"][1, 0] += phi.x0 + at / phi.invDx
        assert oracle.rebox(c.s) == 0
        c.oracle.free(c.o)
        c.o = c.oracle.clone(c.s)
        check(c)
    finally:
        c.close()


# more candidates around a box than the list build stages at once: per-step
# lists of a lattice compressed to 2.5 A, id-keyed skin lists and force-order
# lists of wide boxes (mixed precision: its force-call tolerances)
@pytest.mark.parametrize("precision,edges,bf,lat", [
    (cg.PREC_FP64, (11, 10, 10), 1.0, 2.5), (cg.PREC_FP64, (14, 14, 15), 1.45, None),
    (cg.PREC_MIXED, (14, 14, 15), 1.45, None)])
def test_two_tiles_of_candidates(oracle, precision, edges, bf, lat):
    c = Case(oracle, cg.POT_EAM_TABLE, n=edges, bf=bf, lat=lat, temp=300.0, amp=0.02)
    try:
        assert 27 * c.s.contents.ntot > 900 * c.s.contents.nboxes
        if precision == cg.PREC_FP64:
            check(c)
            return
        c.oracle_force()
        d = c.device(precision)
        assert d.list_info()[0]
        d.force()
        d.download(c.s)
        d.close()
        cmp = compare_forces(c.s, c.o)
        assert cmp["f_rel_rms"] < 1e-5 and cmp["f_max_rel"] < 1e-4, cmp
        assert cmp["rho_max_rel"] < 1e-6 and cmp["fi_max_rel"] < 1e-5, cmp
    finally:
        c.close()
