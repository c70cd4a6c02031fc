"""Batches whose members each fit a cluster of CTAs: MIXED solves are resident up to a few
rounds of clusters and run the multi-kernel CG beyond, FP64 ones are resident in any
number.  The same states either way, bit for bit."""
import numpy as np
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu


def steps(scn, members, precision, resident):
    """Two steps of a batch of copies: the first member's state, and the launches."""
    bs = X.BatchSolver([scn.grid] * members)
    bs.set_option(X.OPT_SMALL_SOLVE, resident)
    bs.upload([scn.copy_state()] * members)
    n0 = X.load().efdc_xm_kernel_launches()
    for n in (1, 2):
        out = bs.step_device([X.make_params(scn.params, n=n, tn=scn.tn(n),
                                            precision=precision)] * members)
        assert all(r.status == X.OK for r in out)
    launches = X.load().efdc_xm_kernel_launches() - n0
    sts = [scn.copy_state() for _ in range(members)]
    bs.download(sts)
    bs.close()
    return sts, launches


# members of one and of several units a CTA; (few rounds, many rounds)
@pytest.mark.parametrize("cells,few,many", [(1100, 64, 1024), (12000, 16, 128), (30000, 8, 96)])
def test_rounds(cells, few, many):
    scn = S.config3_member(1, cells)
    for members, mixed_resident in ((few, True), (many, False)):
        for precision, resident in ((X.PREC_FP64, True), (X.PREC_MIXED, mixed_resident)):
            a, la = steps(scn, members, precision, 1)
            b, lb = steps(scn, members, precision, 0)
            assert (la < lb) if resident else (la == lb), (members, precision, la, lb)
            for m in (0, members // 2, members - 1):
                for k in ("p", "hp", "uhdye", "vhdxe"):
                    np.testing.assert_array_equal(a[m][k], b[m][k], err_msg=f"{m}:{k}")
