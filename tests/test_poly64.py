"""The FP64 Chebyshev kernels at the ends of their polynomial tables, against
the oracle: a lattice of 3.2 A lies inside them; at 2.7 A the nearest pairs
straddle the table's lower end (1.92 A for Cu), at 2.5 A all of them are below
it and the density is past the embedding table's end.  Outside the tables the
kernels sum the series, so the tolerances are those of the FP64 parity tests."""
import pytest

import comd_gb300 as cg
from helpers import Case, compare_forces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lat", [3.2, 2.7, 2.5])
def test_forces_at_the_table_ends(oracle, lat):
    c = Case(oracle, cg.POT_EAM_CHEBY, n=(8, 7, 9), lat=lat, amp=0.05)
    try:
        c.oracle_force()
        d = c.device(cg.PREC_FP64)
        e, stress = d.force()
        d.download(c.s)
        d.close()
        cmp = compare_forces(c.s, c.o)
        assert cmp["f_max_rel"] < 1e-11, cmp
        assert cmp["e_max_rel"] < 1e-11, cmp
        assert cmp["rho_max_rel"] < 1e-12, cmp
        assert cmp["fi_max_rel"] < 1e-12, cmp
        assert abs(e - c.o.contents.e) <= 1e-12 * abs(c.o.contents.e)
        assert abs(stress - c.o.contents.stress) <= 1e-10 * abs(c.o.contents.stress)
    finally:
        c.close()
