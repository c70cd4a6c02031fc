"""efdc_xm_congrad_noalloc where fewer CTAs can be resident together than its launch
has: on a stream that owns part of the GPU's multiprocessors.  The same bits as on the
whole GPU."""
import ctypes as C

import numpy as np
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu


def partition_stream(sms):
    """A stream of a green context of about `sms` multiprocessors."""
    drv = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        if r[0] != drv.CUresult.CUDA_SUCCESS:
            pytest.skip(f"no green contexts here: {r[0]}")
        return r[1] if len(r) == 2 else r[1:]

    dev = ok(drv.cuDeviceGet(0))
    res = ok(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, n, _rest = ok(drv.cuDevSmResourceSplitByCount(1, res, 0, sms))
    assert n == 1
    desc = ok(drv.cuDevResourceGenerateDesc(groups, 1))
    ctx = ok(drv.cuGreenCtxCreate(desc, dev, drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    st = ok(drv.cuGreenCtxStreamCreate(ctx, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))

    def close():
        drv.cuStreamDestroy(st)
        drv.cuGreenCtxDestroy(ctx)

    return int(st), close


# more CTAs than the partition holds with one and with two cells per thread, and a system
# that fits it
@pytest.mark.parametrize("nx,ny", [(300, 240), (420, 330), (40, 30)])
@pytest.mark.parametrize("sms", [8, 40])
def test_partition(nx, ny, sms):
    import torch
    torch.zeros(1, device="cuda")
    stream, close = partition_stream(sms)
    scn = S.make_scenario(nx, ny, seed=41, land_frac=0.05, obc_sides=("W",), amp=0.5, dt=10.0)
    st, g = scn.copy_state(), scn.grid
    sol = X.Solver(g)
    sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1)), st, diag=True)
    sol.close()
    i0 = np.arange(1, scn.la)
    for k, src, nb in (("cce", "ccw", "lec"), ("ccn", "ccs", "lnc")):
        st[k][i0] = np.where(g[nb][i0] <= scn.la, st[src][g[nb][i0] - 1], 0.0)
    t = {k: torch.from_numpy(np.ascontiguousarray(g[k], dtype=np.int32)).cuda()
         for k in ("lnc", "lsc", "lec", "lwc")}
    for k in ("ccc", "ccs", "ccn", "ccw", "cce", "fptmp"):
        t[k] = torch.from_numpy(st[k]).cuda()
    out = []
    for s in (None, stream):
        p = torch.from_numpy(scn.state["p"]).cuda()
        its, rsq = C.c_int32(-1), C.c_double(-1.0)
        torch.cuda.synchronize()
        rc = X.load().efdc_xm_congrad_noalloc(
            scn.la, *(t[k].data_ptr() for k in ("lnc", "lsc", "lec", "lwc", "ccc", "ccs", "ccn",
                                                "ccw", "cce", "fptmp")),
            p.data_ptr(), 1e-10, 500, C.c_void_p(s), C.byref(its), C.byref(rsq))
        torch.cuda.synchronize()
        assert rc == X.OK, X.load().efdc_xm_last_error()
        out.append((its.value, rsq.value, p.cpu().numpy()))
    close()
    assert out[0][:2] == out[1][:2]
    np.testing.assert_array_equal(out[0][2], out[1][2])
