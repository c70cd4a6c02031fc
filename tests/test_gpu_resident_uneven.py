"""Batches of many small members and a few larger ones: no cluster of the largest
member's size for each small one.  What runs instead -- groups of each member's own
size, or the multi-kernel CG -- gives the same states as the multi-kernel CG, bit for
bit."""
import numpy as np
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu


def steps(scns, precision, resident):
    bs = X.BatchSolver([s.grid for s in scns])
    bs.set_option(X.OPT_SMALL_SOLVE, resident)
    sts = [s.copy_state() for s in scns]
    bs.upload(sts)
    n0 = X.load().efdc_xm_kernel_launches()
    for n in (1, 2):
        out = bs.step_device([X.make_params(s.params, n=n, tn=s.tn(n), precision=precision)
                              for s in scns])
        assert all(r.status == X.OK for r in out)
    launches = X.load().efdc_xm_kernel_launches() - n0
    bs.download(sts)
    bs.close()
    return sts, launches


# (small members, larger members, whether they fit the chip together)
@pytest.mark.parametrize("small,large,fit", [((15, 1100), (1, 58000), True),
                                             ((63, 1100), (1, 58000), True),
                                             ((300, 1100), (1, 58000), False),
                                             ((255, 1100), (2, 12000), False)])
@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
def test_uneven(small, large, fit, precision):
    a, b = (S.config3_member(k, n) for k, (_, n) in enumerate((small, large)))
    scns = [a] * (small[0] // 2) + [b] * large[0] + [a] * (small[0] - small[0] // 2)
    sa, la = steps(scns, precision, 1)
    sb, lb = steps(scns, precision, 0)
    assert (la < lb) if fit else (la == lb), (la, lb)
    for m in (0, small[0] // 2, len(scns) - 1):
        for k in ("p", "hp", "uhdye", "vhdxe"):
            np.testing.assert_array_equal(sa[m][k], sb[m][k], err_msg=f"{m}:{k}")
