"""efdc_xm_autotune of a context whose solves are resident: the options of the
multi-kernel iteration, which those solves do not use, are left as they are, and the
measured line is not replayed by a context that runs the multi-kernel iteration."""
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu

KEPT = {X.OPT_KERNEL_VARIANT: ("kernel_variant", 2), X.OPT_CTAS_MATVEC: ("ctas_matvec", 3),
        X.OPT_CTAS_UPDATE: ("ctas_update", 2), X.OPT_GRAPH_ITERS: ("graph_iters", 7)}


@pytest.mark.parametrize("precision", [X.PREC_FP64, X.PREC_MIXED])
def test_resident(tmp_path, precision):
    scn = S.make_scenario(120, 90, seed=5, depth=(4.0, 30.0), amp=0.4, iterm=500,
                          fill_dead_ends=True)
    table = tmp_path / "tune.txt"
    sol = X.Solver(scn.grid)
    for opt, (_, v) in KEPT.items():
        sol.set_option(opt, v)
    sol.step(X.make_params(scn.params, n=1, tn=scn.tn(1), precision=precision), scn.copy_state())
    sch, ms = sol.autotune(precision, table, measure=True)
    assert ms > 0
    for k, v in KEPT.values():
        assert sch[k] == v
    key = sol.tune_key(precision)
    assert X.tune_lookup(table, key) == sch
    sol.set_option(X.OPT_SMALL_SOLVE, 0)
    multi = sol.tune_key(precision)
    assert multi != key and X.tune_lookup(table, multi) is None
    sol.close()
    # a table from before the key told resident solves apart: replayed, without a step
    old = dict(sch, poly_threshold=40)
    table.write_text(table.read_text().replace(key, multi).replace(
        f"poly={sch['poly_threshold']}", "poly=40"))
    sol = X.Solver(scn.grid)
    assert sol.autotune(precision, table) == (old, 0.0)
    sol.close()
