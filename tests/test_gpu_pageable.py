"""Host arrays in pageable memory: small transfers packed, larger ones in pieces
through a page-locked buffer by several threads.  The same steps on page-locked
arrays, on pageable ones and on both kinds in one call give the same states bit for
bit, and leave what a download does not write (L = 1, LC and the element past it)."""
import numpy as np
import pytest
import torch

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu


def basin(nx, ny, seed):
    return S.make_scenario(nx, ny, seed=seed, depth=(4.0, 30.0), corr_len_m=1000.0, amp=0.4,
                           iterm=500, fill_dead_ends=True)


def arrays(scn, kind):
    """The state with its fields in pageable memory, page-locked, or by turns."""
    st = scn.copy_state()
    n = scn.lc + 1
    for i, (k, v) in enumerate(sorted(st.items())):
        if not isinstance(v, np.ndarray) or v.shape != (n,):
            continue
        pin = kind == "locked" or (kind == "both" and i % 2 == 0)
        t = torch.empty(n, dtype=torch.from_numpy(v).dtype, pin_memory=pin).numpy()
        t[:] = v
        if k in ("p", "hp", "uhdye", "vhdxe", "hu"):
            t[[0, scn.lc - 1, scn.lc]] = 7.25
        st[k] = t
    return st


# 31 fields of a state: packed; packed up to the buffer's 4 MiB; pieces, one thread
# and more, with a last piece of a few bytes; several members
@pytest.mark.parametrize("sizes", [[(24, 17)], [(130, 127)], [(140, 133)], [(265, 248)],
                                   [(520, 410)], [(140, 133), (24, 17), (200, 170)]])
def test_same_steps(sizes):
    scns = [basin(nx, ny, 3 + i) for i, (nx, ny) in enumerate(sizes)]
    ref = None
    for kind in ("locked", "pageable", "both"):
        sts = [arrays(s, kind) for s in scns]
        if len(scns) == 1:
            sol = X.Solver(scns[0].grid)
            for n in (1, 2):
                sol.step(X.make_params(scns[0].params, n=n, tn=scns[0].tn(n)), sts[0])
        else:
            sol = X.BatchSolver([s.grid for s in scns])
            sol.upload(sts)
            for n in (1, 2):
                sol.step_device([X.make_params(s.params, n=n, tn=s.tn(n)) for s in scns])
            sol.download(sts)
        sol.close()
        if ref is None:
            ref = sts
            continue
        for a, b in zip(sts, ref):
            for k, v in b.items():
                if isinstance(v, np.ndarray):
                    np.testing.assert_array_equal(a[k], v, err_msg=f"{kind}:{k}")
