"""Contexts created by one host thread while others step theirs for the first time,
which captures the step as a graph: neither is refused, and all step alike."""
import threading

import numpy as np
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu


def test_create_beside_first_steps():
    scn = S.make_scenario(70, 50, seed=3, depth=(4.0, 30.0), amp=0.4, fill_dead_ends=True)
    errors, states = [], []

    def work():
        try:
            for _ in range(25):
                sol, st = X.Solver(scn.grid), scn.copy_state()
                for n in (1, 2):
                    assert sol.step(X.make_params(scn.params, n=n, tn=scn.tn(n)), st).status == X.OK
                sol.close()
                states.append(st)
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(repr(e))

    th = [threading.Thread(target=work) for _ in range(5)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors
    assert len(states) == 125
    for st in states[1:]:
        for k in ("p", "hp", "uhdye", "vhdxe"):
            np.testing.assert_array_equal(st[k], states[0][k], err_msg=k)
