"""The kernels that only large systems reach, at sizes past their lines: the
mixed-precision passes with a thread per atom (Chebyshev from 60,000 atoms,
table from 230,000, LJ from 100,000), their lists whole and overflowed, against
the oracle (LJ's force jumps by 1e-4 Ha/A at the cutoff: atoms with a pair within
2e-6 A of it, ten times the rounding of an FP32 position, are left out); and the adjoint's kernels with four threads an atom (from 12,000)
and one (from 2^19).  The adjoint's sums over a periodic system that is tiled k
times are k times those over one tile: box-relative positions are held to
4e-16 A and the 32nd basis function's slope is 10^3, so to 1e-10 of the largest."""
import numpy as np
import pytest

import comd_gb300 as cg
from comd_gb300.abi import by_id, slot_views
from helpers import Case, compare_forces, world_by_id
from test_fo_lanes import without_last_atom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("potential,edges,cap", [
    (cg.POT_EAM_CHEBY, (25, 26, 24), 0), (cg.POT_EAM_CHEBY, (25, 26, 24), 54),
    (cg.POT_EAM_CHEBY, (25, 26, 24), 8), (cg.POT_EAM_TABLE, (39, 38, 40), 54)])
def test_thread_per_atom(oracle, potential, edges, cap):
    c = Case(oracle, potential, n=edges, bf=1.2, temp=300.0, amp=0.05)
    try:
        without_last_atom(c)
        c.oracle_force()
        d = c.device(cg.PREC_MIXED)
        assert d.list_info()[0]
        if cap:
            d.set_list_capacity(cap)
        e, _ = d.force()
        d.download(c.s)
        d.close()
        n = c.s.contents.ntot
        cmp = compare_forces(c.s, c.o)
        assert cmp["f_rel_rms"] < 1e-5 and cmp["f_max_rel"] < 1e-4, cmp
        assert cmp["e_max_rel"] < 1e-6, cmp
        assert cmp["rho_max_rel"] < 1e-6 and cmp["fi_max_rel"] < 1e-5, cmp
        assert abs(e - c.o.contents.e) < 1e-7 * n
    finally:
        c.close()


@pytest.mark.parametrize("cap", [0, 84])
def test_lj_thread_per_atom(oracle, cap):
    spatial = pytest.importorskip("scipy.spatial")
    c = Case(oracle, cg.POT_LJ, n=(29, 30, 31), bf=1.2, temp=300.0, amp=0.05)
    try:
        without_last_atom(c)
        n = c.s.contents.ntot
        box = np.array(list(c.s.contents.bounds))
        tree = spatial.cKDTree(np.mod(world_by_id(c.s), box), boxsize=box)
        rc = c.s.contents.pot.contents.cutoff
        at = tree.query_pairs(rc + 2e-6, output_type="ndarray")
        inside = tree.query_pairs(rc - 2e-6, output_type="ndarray")
        code = np.setdiff1d(at[:, 0] * n + at[:, 1], inside[:, 0] * n + inside[:, 1])
        sure = np.ones(n, bool)
        sure[code // n] = sure[code % n] = False
        assert sure.mean() > 0.99
        c.oracle_force()
        d = c.device(cg.PREC_MIXED)
        assert d.list_info()[0]
        if cap:
            d.set_list_capacity(cap)
        e, _ = d.force()
        d.download(c.s)
        d.close()
        f, fo = by_id(c.s, "f"), by_id(c.o, "f")
        off, largest = np.abs(f - fo)[sure], np.abs(fo).max(axis=0)
        assert off[:, :3].max() < 1e-4 * largest[:3].max()
        assert np.sqrt((off[:, :3] ** 2).mean()) < 1e-5 * np.sqrt((fo[:, :3] ** 2).mean())
        assert off[:, 3].max() < 1e-6 * largest[3]
        assert abs(e - c.o.contents.e) < 1e-7 * n
    finally:
        c.close()


def tile(c, small, n):
    """c's perfect lattice with the displacements and momenta of small's (n^3
    cells); the id in small of every atom of c"""
    h = 0.5 * small.pot.ptr.contents.lat

    def site(x):  # half-cells from the first atom's sublattice, modulo the tile
        return np.rint((x - first) / h).astype(int) % (2 * n)

    perfect = Case(c.oracle, cg.POT_EAM_CHEBY, n=(n, n, n), amp=0.0, temp=0.0)
    w0 = world_by_id(perfect.s)
    perfect.close()
    first = w0[0]
    shift = world_by_id(small.s) - w0
    shift -= 2 * n * h * np.round(shift / (2 * n * h))
    at = np.full((2 * n,) * 3, -1)
    at[tuple(site(w0).T)] = np.arange(len(w0))
    v = slot_views(c.s)
    occupied = (np.arange(64)[None, :] < v["natoms"][:, None]).reshape(-1)
    w = world_by_id(c.s)
    ids = at[tuple(site(w).T)]
    assert (ids >= 0).all()
    mine = ids[v["id"][occupied]]
    v["r"][occupied] += shift[mine]
    v["p"][occupied] = by_id(small.s, "p")[mine]
    assert c.oracle.rebox(c.s) == 0
    return ids


def gradients(c, target, cap=0):
    d = c.device(cg.PREC_FP64)
    if cap:
        d.set_list_capacity(cap)
    out = [d.energy_grad(), d.force_loss_grad(target), d.traj_energy_grad(2, 1e-15, 1)]
    d.close()
    return out


def same(a, b, factor, tol):
    for (va, ga), (vb, gb) in zip(a, b):
        assert abs(va - factor * vb) <= tol * abs(va)
        for q in range(3):
            s = slice(32 * q, 32 * q + 32)
            assert np.abs(ga[s] - factor * gb[s]).max() <= tol * np.abs(ga[s]).max(), q


@pytest.mark.parametrize("tiles", [(3, 3, 2), (9, 9, 8)])
def test_adjoint_of_a_tiled_system(oracle, tiles):
    n = 6
    small = Case(oracle, cg.POT_EAM_CHEBY, n=(n, n, n), amp=0.05, temp=300.0)
    c = Case(oracle, cg.POT_EAM_CHEBY, n=tuple(n * t for t in tiles), amp=0.0, temp=0.0)
    try:
        ids = tile(c, small, n)
        target = np.random.default_rng(5).normal(0.0, 1e-3, (small.s.contents.ntot, 3))
        same(gradients(c, np.ascontiguousarray(target[ids])), gradients(small, target),
             int(np.prod(tiles)), 1e-10)
    finally:
        c.close()
        small.close()


# overflowed lists: the same pairs by the stencil, summed in another order
@pytest.mark.parametrize("cap", [8, 42])
def test_adjoint_with_overflowed_lists(oracle, cap):
    c = Case(oracle, cg.POT_EAM_CHEBY, n=(6, 7, 6), amp=0.08, temp=600.0)
    try:
        target = np.random.default_rng(5).normal(0.0, 1e-3, (c.s.contents.ntot, 3))
        same(gradients(c, target, cap), gradients(c, target), 1, 1e-10)
    finally:
        c.close()
