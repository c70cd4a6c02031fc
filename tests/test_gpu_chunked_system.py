"""The scaled system (CCC, CCS, CCW, CCE, CCN, FPTMP; calpuv2c.f90:371-399) asked
for after an efdc_xm_step_batch that ran in member chunks: every member's, as after
the same step of all members at once, bit for bit."""
import numpy as np
import pytest

import cases
import efdc_xm as X

pytestmark = pytest.mark.gpu

SYMMETRIC = ("basin_fp64", "tidal_flat_99", "legacy_dry_1")
UNSYMMETRIC = ("basin_fp64", "radiation_all_sides", "radiation_closed_face")


@pytest.mark.parametrize("device_loops", [0, 1])
@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
@pytest.mark.parametrize("names", [SYMMETRIC, UNSYMMETRIC])
def test_system_after_chunks(names, precision, resident, device_loops):
    mem = [cases.build(n)[0] for n in names]
    prm = [X.make_params(m.params, n=1, tn=m.tn(1) * 10.0, precision=precision) for m in mem]
    got = []
    for chunked in (True, False):
        bs = X.BatchSolver([m.grid for m in mem])
        bs.set_option(X.OPT_SMALL_SOLVE, resident)
        bs.set_option(X.OPT_DEVICE_LOOPS, device_loops)
        sts = [m.copy_state() for m in mem]
        if chunked:
            out = bs.step(prm, sts)
        else:
            bs.upload(sts)
            out = bs.step_device(prm)
        assert all(r.status == X.OK for r in out)
        bs.download(sts, diag=True)
        bs.close()
        got.append(sts)
    # without an unsymmetric member the multi-kernel FP64 solve forms no CCE, CCN
    cross = names is UNSYMMETRIC or resident or precision == X.PREC_MIXED
    for m, scn in enumerate(mem):
        for k in ("ccc", "ccs", "ccw", "fptmp") + (("cce", "ccn") if cross else ()):
            a, b = (s[m][k][1:scn.la] for s in got)
            assert np.isfinite(b).all()
            np.testing.assert_array_equal(a, b, err_msg=f"{m}:{k}")
        assert got[0][m]["ccc"][1:scn.la].min() == 1.0  # scaled by the member's minimum
