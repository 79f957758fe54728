"""FP64 with open boundaries: atoms far outside the domain stay in its edge
boxes, where FP32 no longer tells a pair inside the cutoff from one beyond.
Two LJ atoms 1e-6 A inside the cutoff, half an Angstrom (the list build's margin is
for one) to 1e5 A outside the corner box, in one box and in two that share a
face, against the oracle.  At 1e5 A a coordinate is held to 1.5e-11 A, which
changes the energy, about r^-6 there, by 2e-11 of it; bound 1e-10."""
import numpy as np
import pytest

import comd_gb300 as cg
from comd_gb300.abi import slot_views
from helpers import Case

pytestmark = pytest.mark.gpu


def place(c, atoms):
    """(box, box-relative position) of atoms 0, 1, ...: nothing else is left"""
    v = slot_views(c.s)
    v["natoms"][:] = 0
    for i, (b, r) in enumerate(atoms):
        q = b * 64 + v["natoms"][b]
        v["natoms"][b] += 1
        v["id"][q] = i
        v["r"][q, :3] = r
    c.s.contents.ntot = len(atoms)
    c.oracle.free(c.o)
    c.o = c.oracle.clone(c.s)


@pytest.mark.parametrize("out", [0.5, 0.999, 1.001, 3.0, 50.0, 300.0, 2e3, 1e5])
def test_pair_far_outside(oracle, out):
    c = Case(oracle, cg.POT_LJ, n=(8, 8, 8), periodic=False)
    try:
        rc = c.s.contents.pot.contents.cutoff
        width = c.s.contents.boxsize[1]
        assert width > rc
        d = None
        for trial in range(40):
            rng = np.random.default_rng(trial)
            far = -out * rng.uniform(0.97, 1.0)
            a = np.array([far, rng.uniform(0.0, 0.1), far])
            u = np.array([-rng.uniform(0, 1), 1.5, rng.uniform(-1, 1)])
            b = a + u * ((rc - 1e-6) / np.linalg.norm(u))
            other = trial % 2  # in the next box along y, its coordinates relative to it
            if other:
                b[1] -= width
            place(c, [(0, a), (c.s.contents.nbx[0] if other else 0, b)])
            if d is None:
                d = c.device(cg.PREC_FP64)
            else:
                d.upload(c.s)
            c.oracle_force()
            e, _ = d.force()
            assert c.o.contents.e != 0.0
            assert abs(e - c.o.contents.e) <= 1e-10 * abs(c.o.contents.e), trial
        d.close()
    finally:
        c.close()
