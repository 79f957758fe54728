"""The batch autotuner times pass 2's threads per CTA only where a kernel takes
them: a batch whose passes take several threads an atom keeps the default."""
import pytest

import comd_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cg.PREC_MIXED, cg.PREC_FP64])
def test_small_batch_keeps_the_default(precision):
    pot = cg.eam_potential("cu")
    sims = [cg.fcc(n, 6, 6, pot.ptr.contents.lat, 1.0, 1.0, pot) for n in (6, 7)]
    try:
        for _ in range(3):
            t = cg.batch_autotune(sims, cg.opts(cg.POT_EAM_CHEBY, precision, True), (1.0,),
                                  (0.5,), steps=5)
            assert t.pass2_threads == 512
    finally:
        for s in sims:
            cg.free_host(s)
