"""Pageable host arrays through the ring, which a process has once its contexts have
moved some: uploads and downloads move runs of members, whether their arrays lie back to
back or apart.  The same states as from page-locked arrays, bit for bit, and what a
download does not write (L = 1, LC and the element past it) is left."""
import threading

import numpy as np
import pytest
import torch

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu

MARKED = ("p", "hp", "uhdye", "hu", "lopenbcdry")


def members(sizes):
    return [S.make_scenario(nx, ny, seed=3 + i, depth=(4.0, 30.0), corr_len_m=1000.0, amp=0.4,
                            iterm=500, fill_dead_ends=True) for i, (nx, ny) in enumerate(sizes)]


@pytest.fixture(scope="module", autouse=True)
def ring():
    """A context that has moved 200 MB, and stays."""
    scn = members([(600, 500)])[0]
    sol, st = X.Solver(scn.grid), scn.copy_state()
    for _ in range(2):
        sol.upload(st)
        sol.download(st)
    yield
    sol.close()


def arrays(scns, kind):
    """The members' states: page-locked back to back, pageable back to back, some fields
    of either kind, or pageable apart."""
    sizes = [s.lc + 1 for s in scns]
    sts = [dict() for _ in scns]
    for k, v in scns[0].state.items():
        if not isinstance(v, np.ndarray) or v.shape != (sizes[0],):
            for s, st in zip(scns, sts):
                st[k] = s.state[k]
            continue
        pin = kind == "locked" or (kind == "both" and len(k) % 2 == 0)
        t = torch.empty(sum(sizes), dtype=torch.from_numpy(v).dtype, pin_memory=pin)
        o = 0
        for s, st, n in zip(scns, sts, sizes):
            st[k] = np.empty(n, v.dtype) if kind == "apart" else t.numpy()[o:o + n]
            st[k][:] = s.state[k]
            o += n
    return sts


# 64 short members, 600 KB an array (two pieces); members of several pieces and of a part
# of one, at odd offsets
SIZES = [[(44, 28)] * 60 + [(43, 29), (20, 6), (33, 17), (45, 27)],
         [(300, 261), (24, 17), (411, 173), (9, 8), (97, 70)],
         [(140, 133)], [(265, 248)], [(520, 410)]]


@pytest.mark.parametrize("sizes", SIZES)
def test_members(sizes):
    scns = members(sizes)
    ref, moved = None, []
    for kind in ("locked", "back to back", "both", "apart"):
        sts = arrays(scns, kind)
        bs = X.BatchSolver([s.grid for s in scns])
        bs.upload(sts)
        bs.download(sts)
        b0 = X.transfer_bytes()
        bs.upload(sts)
        for n in (1, 2):
            out = bs.step_device([X.make_params(s.params, n=n, tn=s.tn(n)) for s in scns])
            assert all(r.status == X.OK for r in out)
        for s, st in zip(scns, sts):
            for k in MARKED:
                st[k][[0, s.lc - 1, s.lc]] = 7
        bs.download(sts)
        moved.append([a - b for a, b in zip(X.transfer_bytes(), b0)])
        bs.close()
        if ref is None:
            ref = sts
            continue
        for m, (a, b) in enumerate(zip(sts, ref)):
            for k, v in b.items():
                if isinstance(v, np.ndarray):
                    np.testing.assert_array_equal(a[k], v, err_msg=f"{kind}:{m}:{k}")
    # a run of members moves as one range of the staging buffer, the element between two
    # of them with it (a download's without the ghost elements at its ends); a piece may
    # end between two members
    for up, down in moved[1:]:
        assert abs(up - moved[0][0]) <= 8 * 64 and abs(down - moved[0][1]) <= 8 * 64 * 4


def test_threads():
    """More host threads than rings, a context each: some transfers go through the
    driver."""
    scn = members([(265, 248)])[0]
    got = [None] * 6

    def work(i):
        sol, st = X.Solver(scn.grid), scn.copy_state()
        for n in range(1, 7):
            r = sol.step(X.make_params(scn.params, n=n, tn=scn.tn(n)), st)
            assert r.status == X.OK
        sol.close()
        got[i] = st

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(got))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for st in got[1:]:
        for k, v in got[0].items():
            if isinstance(v, np.ndarray):
                np.testing.assert_array_equal(st[k], v, err_msg=k)
