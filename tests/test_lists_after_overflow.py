"""A trajectory that a full box stops (COMDGB_ERR_MAXATOMS, -11) leaves a layout
without the atom that did not fit, and skin lists built from it.  A state
uploaded after that, near enough for the skin test to pass, must not be
computed with those lists: the same forces as a new handle's, to rounding."""
import numpy as np
import pytest

import comd_gb300 as cg
from comd_gb300.abi import by_id, slot_views
from helpers import Case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,steps", [(cg.PREC_FP64, 0), (cg.PREC_FP64, 1),
                                             (cg.PREC_FP64, 3), (cg.PREC_MIXED, 1),
                                             (cg.PREC_MIXED, 3)])
def test_lists_are_built_again(oracle, precision, steps):
    # 3 x 3 x 3 boxes; box 2 holds 63 atoms, and an atom of box 5, above it along
    # y, is about to enter it at 0.2 A a half step
    c = Case(oracle, cg.POT_EAM_CHEBY, n=(7, 7, 7), bf=1.6, amp=0.02, temp=0.0)
    try:
        v = slot_views(c.s)
        assert list(c.s.contents.nbx) == [3, 3, 3] and v["natoms"][2] == 63
        q = 5 * 64 + int(np.argmin(v["r"][5 * 64:5 * 64 + v["natoms"][5], 1]))
        v["r"][q, 1] = 0.1
        d = c.device(precision)
        persistent, skin, _ = d.list_info()
        assert persistent and skin == 0.5
        e0, _ = d.force()
        d.download(c.s)
        f0 = by_id(c.s, "f")
        # dr = (dt / 2) p / m, dt of 1 fs and m in the reference's units
        dt, m = 1e-15 * 0.529 / 2.418e-17, 1822.83 * c.pot.ptr.contents.mass
        v["p"][q, 1] = -0.2 * m / (dt / 2)
        d.upload(c.s)
        with pytest.raises(cg.ComdgbError) as err:
            if steps:
                d.steps(steps, 1e-15)
            else:
                d.traj_energy_grad(2, 1e-15, 2)
        assert err.value.code == -11
        d.upload(c.s)
        e, _ = d.force()
        d.download(c.s)
        d.close()
        f = by_id(c.s, "f")
        assert abs(e - e0) <= 1e-12 * abs(e0)
        tol = 1e-12 if precision == cg.PREC_FP64 else 1e-5
        assert np.abs(f - f0).max() <= tol * np.abs(f0).max()
    finally:
        c.close()

