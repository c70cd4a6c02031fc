"""efdc_xm_time_kernels after a step whose solve was resident: that solve forms no
operator for the multi-kernel iteration in memory, so the call forms it."""
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
@pytest.mark.parametrize("kw", [{}, {"ispb": 1, "obc_sides": ("W", "E")}])
def test_time_kernels(precision, kw):
    scn = S.make_scenario(120, 90, seed=5, depth=(4.0, 30.0), amp=0.4, iterm=500,
                          fill_dead_ends=True, **kw)
    sol = X.Solver(scn.grid)
    st = scn.copy_state()
    sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1), precision=precision), st)
    kt = sol.time_kernels(precision, 5)  # raises where the iteration stops early
    assert kt.ms_matvec > 0 and kt.ms_update > 0
    sol.close()
