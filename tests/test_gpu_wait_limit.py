"""Waits between the CTAs of a solve that run out (efdc_xm_set_wait_limit): a call
returns EFDC_XM_DEVICE_TIMEOUT unless its results are those of a call that waits as
long as it takes, and the next call with the default limit gives these results.
CONGRAD without allocation looks for the others a few times only, so that some of its
CTAs may come through an exchange; a context's solve waits in vain."""
import numpy as np
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu

LIMITS = [0] * 6 + [1, 2, 4, 8] * 4


@pytest.fixture(autouse=True)
def default_limit():
    yield
    X.set_wait_limit()


def system(nx, ny):
    scn = S.make_scenario(nx, ny, seed=41, obc_sides=("W",), amp=0.5, dt=10.0)
    st, g = scn.copy_state(), scn.grid
    sol = X.Solver(g)
    sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1)), st, diag=True)
    i0 = np.arange(1, scn.la)
    for k, src, nb in (("cce", "ccw", "lec"), ("ccn", "ccs", "lnc")):
        st[k][i0] = np.where(g[nb][i0] <= scn.la, st[src][g[nb][i0] - 1], 0.0)
    return scn, st, sol


def check(call, limits=LIMITS):
    """call() -> (status, results)."""
    rc0, want = call()
    assert rc0 in (X.OK, X.CG_MAXITER)
    seen = []
    for limit in limits:
        old = X.set_wait_limit(limit)
        rc, got = call()
        assert X.set_wait_limit(old) == limit
        seen.append(rc)
        if rc != X.DEVICE_TIMEOUT:
            assert rc == rc0
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
        rc, got = call()
        assert rc == rc0
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
    assert X.DEVICE_TIMEOUT in seen  # CTAs that look once cannot all find the others


@pytest.mark.parametrize("iterm", [1, 500])
def test_noalloc(iterm):
    import torch
    scn, st, sol = system(300, 250)
    sol.close()
    t = {k: torch.from_numpy(np.ascontiguousarray(scn.grid[k], dtype=np.int32)).cuda()
         for k in ("lnc", "lsc", "lec", "lwc")}
    for k in ("ccc", "ccs", "ccn", "ccw", "cce", "fptmp"):
        t[k] = torch.from_numpy(st[k]).cuda()

    def call():
        p = torch.from_numpy(scn.state["p"]).cuda()
        torch.cuda.synchronize()
        rc = X.load().efdc_xm_congrad_noalloc(
            scn.la, *(t[k].data_ptr() for k in ("lnc", "lsc", "lec", "lwc", "ccc", "ccs", "ccn",
                                                "ccw", "cce", "fptmp")),
            p.data_ptr(), 1e-10, iterm, None, None, None)
        return rc, (p.cpu().numpy(),)

    check(call)


def large():
    """A context whose member takes more CTAs than a cluster holds.  MIXED: one
    preconditioner (else each solve's choice follows from the iterations of the last)."""
    scn, st, sol = system(520, 515)
    sol.set_option(X.OPT_POLY_THRESHOLD, 0)
    return scn, st, sol


@pytest.mark.parametrize("iterm", [1, 500])
@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
def test_congrad(precision, iterm):
    scn, st, sol = large()

    def call():
        p = scn.state["p"].copy()
        args = (st["ccc"], st["ccs"], st["ccn"], st["ccw"], st["cce"], st["ccc"], st["fptmp"], p)
        rc, it, rsq = sol.congrad(*args, 1e-10, iterm, precision)
        return rc, (p, it, rsq)

    check(call, [0, 8])
    sol.close()


@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
def test_step(precision):
    scn, _, sol = large()

    def call():
        st = scn.copy_state()
        try:
            r = sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1), precision=precision), st)
        except RuntimeError as e:
            assert "DEVICE_TIMEOUT" in str(e)
            return X.DEVICE_TIMEOUT, ()
        return r.status, (st["p"], st["hp"], st["uhdye"])

    check(call, [0, 8])
    sol.close()


def test_no_further_sweeps():
    """A wetting and drying step (three or four solves) whose first solve runs out of
    time ends with its sweep, and the next one is as if it had not been."""
    scn = S.tidal_flat(n=280, seed=13, dt=5.0)
    sol = X.Solver(scn.grid)
    sweeps, states = [], []
    for limit in (-1, 0, 0, 0, -1):
        X.set_wait_limit(limit)
        st, n0 = scn.copy_state(), X.load().efdc_xm_kernel_launches()
        try:
            r = sol.step(X.make_params(scn.params, n=1, tn=1200.0), st)
            assert r.status == X.OK and r.solves >= 2
            states.append(st)
        except RuntimeError as e:
            assert "DEVICE_TIMEOUT" in str(e)
        sweeps.append(X.load().efdc_xm_kernel_launches() - n0)
    sol.close()
    assert len(states) == 2 and sweeps[0] == sweeps[4] > max(sweeps[1:4])
    for k in ("p", "hp", "uhdye", "lmaskdry"):
        np.testing.assert_array_equal(states[0][k], states[1][k], err_msg=k)
