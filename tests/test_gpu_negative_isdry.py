"""ISDRY < 0: no wetting and drying, and P keeps the solver's value (CALPUV2C
refreshes it from HP for ISDRY = 0 only, calpuv2c.f90:893-897); the depth of an
open-boundary cell is its elevation's (:489-490).  Against the oracle."""
import pytest

import cases
import efdc_xm as X
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_loops", [0, 1])
@pytest.mark.parametrize("name", ["basin_fp64", "radiation_all_sides"])
def test_open_boundary_depths(name, device_loops):
    scn, _, dtn = cases.build(name)
    prm = dict(scn.params, isdry=-1)
    sol, orc = X.Solver(scn.grid), O.Oracle(scn.grid)
    sol.set_option(X.OPT_DEVICE_LOOPS, device_loops)
    a, b = scn.copy_state(), scn.copy_state()
    for n in range(1, 6):
        p = X.make_params(prm, n=n, tn=scn.tn(n) * dtn)
        sa, sb = sol.step(p, a), orc.step(p, b)
        assert sa.status == sb.status == X.OK
    sol.close()
    for k in ("p", "hp", "hu", "hv"):
        assert cases.state_err(a, b, scn.la, k) <= 1e-10, k
