"""Pairs that the FP64 passes' integers do not serve, against the oracle: atoms
at one place (an infinite LJ energy, COMDGB_ERR_NONFINITE, -35; EAM forces that are not
numbers), atoms closer than the range of the integers begins (0.5 A for the Cu
potentials), a pair at exactly the cutoff, whose distance the reference's rounding
decides, and differences of zero, which give forces of zero.  The distances are
formed operation by operation as the oracle forms them, so the tolerances are
those of the FP64 parity tests."""
import numpy as np
import pytest

import comd_gb300 as cg
from comd_gb300.abi import by_id, slot_views
from helpers import Case, LJ_EPS, LJ_MASS, LJ_SIGMA, compare_forces

pytestmark = pytest.mark.gpu


def put(c, d):
    """the first box's second atom at the first one's place plus d"""
    v = slot_views(c.s)
    assert v["natoms"][0] > 1
    v["r"][1] = v["r"][0]
    v["r"][1, :3] += d
    assert c.oracle.rebox(c.s) == 0
    c.oracle.free(c.o)
    c.o = c.oracle.clone(c.s)
    return list(v["id"][:2])


def pair_alone(oracle, d, cutoff=None, potential=cg.POT_LJ):
    """two atoms d apart along x, the first at a corner of the first box"""
    c = Case(oracle, potential, n=(7, 7, 8))
    if cutoff is not None:
        oracle.free(c.o)
        c.pot = cg.lj_potential(LJ_SIGMA, LJ_EPS, cutoff, LJ_MASS)
        c.s = cg.fcc(7, 7, 8, 3.615, 1.0, 1.0, c.pot)
        c.o = oracle.clone(c.s)
    v = slot_views(c.s)
    v["natoms"][1:] = 0
    v["natoms"][0] = c.s.contents.ntot = 2
    v["id"][:2] = [0, 1]
    v["r"][:2] = 0.0
    v["r"][1, 0] = d
    oracle.free(c.o)
    c.o = oracle.clone(c.s)
    return c


@pytest.mark.parametrize("precision", [cg.PREC_FP64, cg.PREC_MIXED])
def test_lj_atoms_at_one_place(oracle, precision):
    c = Case(oracle, cg.POT_LJ, n=(7, 7, 8), temp=300.0)
    try:
        put(c, [0.0, 0.0, 0.0])
        d = c.device(precision)
        with pytest.raises(cg.ComdgbError) as e:
            d.force()
        assert e.value.code == -35
        d.close()
    finally:
        c.close()


@pytest.mark.parametrize("potential", [cg.POT_EAM_TABLE, cg.POT_EAM_CHEBY])
def test_eam_atoms_at_one_place(oracle, potential):
    c = Case(oracle, potential, n=(6, 6, 7), temp=300.0)
    try:
        two = put(c, [0.0, 0.0, 0.0])
        c.oracle_force()
        d = c.device(cg.PREC_FP64)
        d.force()
        d.download(c.s)
        d.close()
        f, fo = by_id(c.s, "f"), by_id(c.o, "f")
        assert np.isnan(fo[two, :3]).all()
        assert np.array_equal(np.isnan(f), np.isnan(fo))
        rest = ~np.isnan(fo)
        assert np.abs(f - fo)[rest].max() < 1e-11 * np.abs(fo[rest]).max()
    finally:
        c.close()


@pytest.mark.parametrize("potential", [cg.POT_EAM_TABLE, cg.POT_EAM_CHEBY, cg.POT_LJ])
@pytest.mark.parametrize("r", [0.6, 0.4999, 0.3, 0.03, 1e-3, 1e-6])
def test_close_pair(oracle, potential, r):
    c = Case(oracle, potential, n=(7, 7, 8), temp=300.0, amp=0.03)
    try:
        put(c, np.array([1.0, -2.0, 2.0]) * (r / 3.0))
        c.oracle_force()
        d = c.device(cg.PREC_FP64)
        e, _ = d.force()
        w, _, _ = d.virial()
        d.download(c.s)
        d.close()
        cmp = compare_forces(c.s, c.o)
        assert cmp["f_max_rel"] < 1e-11 and cmp["e_max_rel"] < 1e-11, cmp
        if potential != cg.POT_LJ:
            assert cmp["rho_max_rel"] < 1e-12 and cmp["fi_max_rel"] < 1e-12, cmp
        assert abs(e - c.o.contents.e) <= 1e-12 * abs(c.o.contents.e)
        wo, _, _ = oracle.virial(c.o, c.kind)
        assert np.abs(w - wo).max() <= 1e-11 * np.abs(wo).max()
    finally:
        c.close()


# cutoffs whose square FP64 rounds down (3.7, 4.7), up (3.9, 4.1) and holds (4.0)
@pytest.mark.parametrize("cutoff", [3.7, 3.9, 4.0, 4.1, 4.7])
def test_pair_at_the_cutoff(oracle, cutoff):
    c = pair_alone(oracle, cutoff, cutoff)
    try:
        c.oracle_force()
        assert c.o.contents.e != 0.0
        d = c.device(cg.PREC_FP64)
        e, _ = d.force()
        assert d.pair_count() == 1
        d.download(c.s)
        d.close()
        assert abs(e - c.o.contents.e) <= 1e-12 * abs(c.o.contents.e)
        assert compare_forces(c.s, c.o)["f_max_rel"] < 1e-12
    finally:
        c.close()


@pytest.mark.parametrize("potential", [cg.POT_EAM_TABLE, cg.POT_EAM_CHEBY, cg.POT_LJ])
def test_no_force_across_a_plane(oracle, potential):
    c = pair_alone(oracle, 2.6, potential=potential)
    try:
        d = c.device(cg.PREC_FP64)
        d.force()
        d.download(c.s)
        d.close()
        f = by_id(c.s, "f")
        assert (f[:, 0] != 0.0).all() and (f[:, 1:3] == 0.0).all()
    finally:
        c.close()
