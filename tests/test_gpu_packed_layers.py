"""Small transfers of more arrays than one launch's job table holds: the explicit
momentum terms of a small basin with many layers.  In a few link operations, as with
few layers, and with the results of the oracle."""
import numpy as np
import pytest

import efdc_xm as X
import oracle as O
import scenario as S

pytestmark = pytest.mark.gpu

SUMS, LAYER = ("fcaxe", "fcaye", "fxe", "fye"), ("fcax", "fcay", "fx", "fy", "cac")


# 4 KC + 6 arrays up, 5 KC + 4 down: below, at and above one table, and more than a call
# moves in one go
@pytest.mark.parametrize("kc", [8, 12, 13, 16, 24, 25])
def test_explicit(kc):
    scn = S.make_scenario(24, 17, seed=3, depth=(4.0, 30.0), amp=0.4, fill_dead_ends=True)
    S.add_momentum(scn, kc=kc, seed=3)
    sol, orc = X.Solver(scn.grid), O.Oracle(scn.grid)
    sol.set_momentum(scn.momentum)
    orc.set_momentum(scn.momentum)
    sol.upload(scn.copy_state())
    a, b = S.momentum_fields(scn, seed=3), S.momentum_fields(scn, seed=3)
    prm = X.make_explicit_params(1.0, 1, 0)
    for _ in range(2):
        n0 = X.transfer_bytes()
        sol.explicit(prm, a)
        up, down = (x - y for x, y in zip(X.transfer_bytes(), n0))
        # packed arrays move at the staging stride, LC + 1 elements
        stride = 8 * (scn.lc + 1)
        assert up % stride == 0 and up // stride >= 4 * kc
        assert down % stride == 0 and down // stride >= 5 * kc
        assert orc.explicit(prm, b) == 0
    sol.close()
    for k in SUMS:
        np.testing.assert_array_equal(a[k][1:scn.la], b[k][1:scn.la], err_msg=k)
    for k in LAYER:
        np.testing.assert_array_equal(a[k][:, 1:scn.la], b[k][:, 1:scn.la], err_msg=k)
