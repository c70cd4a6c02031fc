"""efdc_xm_congrad_noalloc at the sizes where its launch changes: less than a CTA,
the edge of a CTA, and either side of 1, 2 and 4 cells per thread (all-water
basins), against the context's CONGRAD: the same iterations, the surface within
1e-9 m."""
import ctypes as C

import numpy as np
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(5, 4), (32, 16), (33, 16), (296, 256), (297, 256), (592, 256),
                                   (593, 256), (592, 512), (593, 512)])
def test_sizes(nx, ny):
    import torch
    scn = S.make_scenario(nx, ny, seed=41, land_frac=0.0, obc_sides=("W",), amp=0.5, dt=10.0)
    st, g = scn.copy_state(), scn.grid
    sol = X.Solver(g)
    sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1)), st, diag=True)
    i0 = np.arange(1, scn.la)
    for k, src, nb in (("cce", "ccw", "lec"), ("ccn", "ccs", "lnc")):
        st[k][i0] = np.where(g[nb][i0] <= scn.la, st[src][g[nb][i0] - 1], 0.0)
    ref = scn.state["p"].copy()
    rc, it_ref, _ = sol.congrad(st["ccc"], st["ccs"], st["ccn"], st["ccw"], st["cce"], st["ccc"],
                                st["fptmp"], ref, 1e-10, 500)
    sol.close()
    assert rc == X.OK
    t = {k: torch.from_numpy(np.ascontiguousarray(g[k], dtype=np.int32)).cuda()
         for k in ("lnc", "lsc", "lec", "lwc")}
    for k in ("ccc", "ccs", "ccn", "ccw", "cce", "fptmp"):
        t[k] = torch.from_numpy(st[k]).cuda()
    p = torch.from_numpy(scn.state["p"].copy()).cuda()
    its, rsq = C.c_int32(-1), C.c_double(-1.0)
    torch.cuda.synchronize()
    rc = X.load().efdc_xm_congrad_noalloc(
        scn.la, *(t[k].data_ptr() for k in ("lnc", "lsc", "lec", "lwc", "ccc", "ccs", "ccn", "ccw",
                                            "cce", "fptmp")),
        p.data_ptr(), 1e-10, 500, None, C.byref(its), C.byref(rsq))
    assert rc == X.OK
    assert abs(its.value - it_ref) <= 1 and rsq.value <= 1e-10
    assert np.abs(p.cpu().numpy() - ref)[1:scn.la].max() / S.G < 1e-9
