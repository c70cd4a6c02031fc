"""Back-substitution and continuity in one kernel (contexts of up to a tile per CTA) and
in two: a member gives the same bits in a context of its own and in a batch that is
past the line, with open boundaries of every kind, without and with wetting and drying,
and with three time levels."""
import numpy as np
import pytest

import cases
import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu

FIELDS = ("p", "hp", "hu", "hv", "uhdye", "vhdxe", "uhe", "vhe", "sub", "svb", "lmaskdry")


def filler(n):
    return S.make_scenario(n, n, seed=9, depth=(4.0, 30.0), corr_len_m=1000.0, amp=0.4,
                           iterm=500, fill_dead_ends=True)


def run(scns, params, steps=5):
    bs = X.BatchSolver([s.grid for s in scns])
    sts = [s.copy_state() for s in scns]
    bs.upload(sts)
    n0 = X.load().efdc_xm_kernel_launches()
    for n in range(1, steps + 1):
        out = bs.step_device([X.make_params(p, n=n, tn=s.tn(n) * 20.0)
                              for s, p in zip(scns, params)])
        assert all(r.status in (X.OK, X.NEG_DEPTH) for r in out)
    launches = X.load().efdc_xm_kernel_launches() - n0
    bs.download(sts)
    bs.close()
    return sts, launches


@pytest.mark.parametrize("name,isdry", [("radiation_all_sides", 0), ("noise_forcing", 0),
                                        ("noise_forcing", -1), ("tidal_flat_99", 99),
                                        ("legacy_dry_1", 1)])
def test_member_alone_and_in_a_batch(name, isdry):
    scn, big = cases.build(name)[0], filler(420)
    prm = dict(scn.params, isdry=isdry)
    a, _ = run([scn], [prm])
    b, _ = run([big, scn], [big.params, prm])
    for k in FIELDS:
        np.testing.assert_array_equal(a[0][k], b[1][k], err_msg=k)


def test_three_levels():
    scn, big = cases.build("noise_forcing")[0], filler(420)
    for s in (scn, big):
        S.add_three_levels(s)
    lv = dict(tl3_istl=3, nctbc=1, rold=0.0, rnew=1.0)
    a, _ = run([scn], [dict(scn.params, **lv)])
    b, _ = run([big, scn], [dict(big.params, **lv), dict(scn.params, **lv)])
    for k in ("p", "hp", "uhdye", "vhdxe", "uhdy1e", "h2p"):
        np.testing.assert_array_equal(a[0][k], b[1][k], err_msg=k)


def test_line():
    """One launch more per step past a tile per CTA."""
    _, small = run([filler(100)], [filler(100).params])
    _, large = run([filler(700)], [filler(700).params])
    assert large == small + 5
