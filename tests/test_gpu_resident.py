"""Resident solves (EFDC_XM_OPT_SMALL_SOLVE): the whole solve of a member in one
launch, its vectors on the chip, against the multi-kernel CG of the same
context, bit for bit -- states, CG iterations, refinement passes.

Sizes at which the launch changes its form: a member of one 4-tile unit (no
exchange between CTAs), ragged last units, one, two, four and eight units per CTA, and
batches that take several launches; with radiation boundaries (the four-array
operator), wetting and drying, three time levels, the standalone CONGRAD and
the adjoint's solve.
"""
import numpy as np
import pytest

import cases
import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu

FIELDS = ("p", "hp", "hu", "hv", "uhdye", "vhdxe", "sub", "svb", "lmaskdry")


def basin(nx, ny, seed=5, **kw):
    kw.setdefault("explicit_noise", 1e-4)
    return S.make_scenario(nx, ny, seed=seed, depth=(4.0, 30.0), corr_len_m=1000.0, amp=0.4,
                           iterm=500, fill_dead_ends=True, **kw)


def run(mem, resident, precision, steps, device_loops=1, poly=None):
    bs = X.BatchSolver([m.grid for m in mem])
    bs.set_option(X.OPT_SMALL_SOLVE, resident)
    bs.set_option(X.OPT_DEVICE_LOOPS, device_loops)
    if poly is not None:
        bs.set_option(X.OPT_POLY_THRESHOLD, poly)
    sts = [m.copy_state() for m in mem]
    bs.upload(sts)
    its = []
    for n in range(1, steps + 1):
        out = bs.step_device([X.make_params(m.params, n=n, tn=m.tn(n), precision=precision)
                              for m in mem])
        assert all(r.status in (X.OK, X.NEG_DEPTH) for r in out), [r.as_dict() for r in out]
        its.append([(r.status, r.iters_total, r.solves, r.outer_refinements, r.rsq_last)
                    for r in out])
    bs.download(sts)
    bs.close()
    return sts, its


def same(mem, precision, steps=3, **kw):
    a, ia = run(mem, 1, precision, steps, **kw)
    b, ib = run(mem, 0, precision, steps, **kw)
    assert ia == ib
    for m in range(len(mem)):
        for k in FIELDS:
            np.testing.assert_array_equal(a[m][k], b[m][k], err_msg=f"{m}:{k}")


SIZES = [(20, 6), (33, 17), (64, 16), (97, 70), (200, 120), (250, 190), (300, 211), (520, 515),
         (640, 530), (830, 801)]


@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_one_basin(nx, ny, precision):
    same([basin(nx, ny)], precision)


@pytest.mark.parametrize("poly", [0, 100000])
def test_mixed_preconditioners(poly):
    same([basin(150, 90)], X.PREC_MIXED, poly=poly)


@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
@pytest.mark.parametrize("device_loops", [0, 1])
def test_forms(precision, device_loops):
    """Radiation on all sides, an unsymmetric operator, wetting and drying, alone
    and as one batch with a plain basin."""
    mem = [cases.build(n)[0] for n in ("radiation_all_sides", "radiation_closed_face",
                                       "tidal_flat_99", "legacy_dry_1", "basin_fp64")]
    for m in mem:
        same([m], precision, 6, device_loops=device_loops)
    same(mem, precision, 6, device_loops=device_loops)


@pytest.mark.parametrize("names", [("radiation_all_sides", "legacy_dry_1"),
                                   ("radiation_closed_face", "tidal_flat_99")])
def test_four_rows_of_quads(names):
    """The FP64 form of members of more than 592 units, which reads the operator in
    each iteration: small members with both operators beside a basin that takes it,
    and (two launches) beside two."""
    small = [cases.build(n)[0] for n in names]
    same([basin(830, 801)] + small, X.PREC_FP64)
    same(small + [basin(1010, 640, seed=k) for k in (3, 4)], X.PREC_FP64, 2)


@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
def test_several_launches(precision):
    """More members than one launch holds: 6 of about 200 units, and small ones."""
    mem = [basin(450, 440, seed=k) for k in range(6)] + [basin(40, 30, seed=9)]
    same(mem, precision, 2)


@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
def test_congrad(precision):
    """The standalone solve against the multi-kernel one."""
    scn = basin(90, 75)
    sol = X.Solver(scn.grid)
    st = scn.copy_state()
    sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1)), st, diag=True)
    g = scn.grid  # a symmetric operator's CCE, CCN are not formed by a step
    i0 = np.arange(1, scn.la)
    for k, src, nb in (("cce", "ccw", "lec"), ("ccn", "ccs", "lnc")):
        st[k][i0] = np.where(g[nb][i0] <= scn.la, st[src][g[nb][i0] - 1], 0.0)
    out = []
    for resident in (1, 0):
        sol.set_option(X.OPT_SMALL_SOLVE, resident)
        p = scn.state["p"].copy()
        rc, it, rsq = sol.congrad(st["ccc"], st["ccs"], st["ccn"], st["ccw"], st["cce"],
                                  st["ccc"], st["fptmp"], p, 1e-12, 500, precision)
        out.append((rc, it, rsq, p))
    sol.close()
    assert out[0][:3] == out[1][:3] and out[0][0] == X.OK
    np.testing.assert_array_equal(out[0][3], out[1][3])


def test_failures_and_empty_solves():
    """ITERM reached, a NaN right-hand side, and a state at rest (RPCG = 0)."""
    for resident in (1, 0):
        scn = basin(90, 75)
        sol = X.Solver(scn.grid)
        sol.set_option(X.OPT_SMALL_SOLVE, resident)
        r = sol.step(X.make_params(dict(scn.params, iterm=1), n=1, tn=scn.tn(1)),
                     scn.copy_state())
        assert r.status == X.CG_MAXITER and r.iters_total == 1
        bad = scn.copy_state()
        bad["qsume"][100] = np.nan
        for precision in (X.PREC_FP64, X.PREC_MIXED):
            r = sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1), precision=precision), bad)
            assert r.status == X.NONFINITE
            good = scn.copy_state()
            r = sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1), precision=precision), good)
            assert r.status == X.OK
        sol.close()
        rest = S.make_scenario(60, 40, seed=2, obc_sides=(), manning=0.0)
        sol = X.Solver(rest.grid)
        sol.set_option(X.OPT_SMALL_SOLVE, resident)
        r = sol.step(X.make_params(rest.params, n=1, tn=rest.tn(1)), rest.copy_state())
        assert r.status == X.OK and r.iters_total == 0
        sol.close()


def test_two_contexts_in_two_threads():
    """Two host threads, a context each, whose resident launches each fill the GPU."""
    import threading
    scn = basin(520, 515)
    ref, _ = run([scn], 1, X.PREC_FP64, 20)
    got = [None, None]

    def work(i):
        got[i] = run([scn], 1, X.PREC_FP64, 20)[0]

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for g in got:
        for k in FIELDS:
            np.testing.assert_array_equal(g[0][k], ref[0][k])
