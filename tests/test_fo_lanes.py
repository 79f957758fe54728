"""The mixed-precision passes with several threads per atom, against the
oracle: at sizes either side of the lines between eight, four, two threads
and one (Chebyshev 12,000 and 60,000 atoms, table 24,000, 140,000 and
230,000, LJ 24,000 and 100,000), with an atom taken out so that the atoms do
not fill the last warp.  Force calls to the mixed-precision tolerances; ten
steps, whose update the lanes share, to what those force errors come to: a
force off by 1e-5 of the largest (below 0.1 Ha/A) moves an atom of 1.2e5 m_e
by less than 1e-8 A in 10 fs, the positions' tolerance is 1e-6 A."""
import numpy as np
import pytest

import comd_gb300 as cg
from comd_gb300.abi import slot_views
from helpers import Case, compare_forces, world_by_id

pytestmark = pytest.mark.gpu


def without_last_atom(c):
    """removes the atom of the largest id from the case's host simulation"""
    s = c.s.contents
    v = slot_views(c.s)
    last = s.ntot - 1
    slot = next(int(q) for q in np.flatnonzero(v["id"] == last) if q % 64 < v["natoms"][q // 64])
    b = slot // 64
    end = b * 64 + v["natoms"][b] - 1
    for name in ("id", "iType", "mass", "r", "p", "f", "rho", "fi"):
        v[name][slot] = v[name][end]
    v["natoms"][b] -= 1
    s.ntot -= 1
    c.oracle.free(c.o)
    c.o = c.oracle.clone(c.s)


@pytest.mark.parametrize("potential,edges", [
    (cg.POT_EAM_CHEBY, (6, 7, 6)), (cg.POT_EAM_CHEBY, (15, 14, 16)),
    (cg.POT_EAM_TABLE, (7, 6, 8)), (cg.POT_EAM_TABLE, (19, 18, 20)),
    (cg.POT_EAM_TABLE, (34, 33, 35)), (cg.POT_EAM_TABLE, (39, 38, 40)),
    (cg.POT_LJ, (8, 7, 9)), (cg.POT_LJ, (19, 18, 20))])
def test_lanes(oracle, potential, edges):
    c = Case(oracle, potential, n=edges, bf=1.2, temp=300.0, amp=0.05)
    try:
        without_last_atom(c)
        c.oracle_force()
        d = c.device(cg.PREC_MIXED)
        assert d.list_info()[0]
        e, _ = d.force()
        d.download(c.s)
        n = c.s.contents.ntot
        cmp = compare_forces(c.s, c.o)
        assert cmp["f_rel_rms"] < 1e-5 and cmp["f_max_rel"] < 1e-4, cmp
        assert cmp["e_max_rel"] < 1e-6, cmp
        if potential != cg.POT_LJ:
            assert cmp["rho_max_rel"] < 1e-6 and cmp["fi_max_rel"] < 1e-5, cmp
        assert abs(e - c.o.contents.e) < 1e-7 * n
        if potential != cg.POT_LJ and n < 100000:
            d.steps(10, 1e-15)
            d.download(c.s)
            assert c.oracle.steps(c.o, 10, 1e-15, c.kind) == 0
            dx = world_by_id(c.s) - world_by_id(c.o)
            box = np.array(list(c.s.contents.bounds))
            dx -= box * np.round(dx / box)
            assert np.abs(dx).max() < 1e-6
        d.close()
    finally:
        c.close()
