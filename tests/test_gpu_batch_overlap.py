"""A chunked efdc_xm_step_batch whose chunks really overlap: page-locked host
arrays, members large enough for a chunk's copies to take longer than a step,
and a second context (no first-use delays).  The arrays of 4-byte elements
(LOPENBCDRY) go up while the 8-byte arrays of earlier members come down; a
member's range of one must not touch another member's range of the other."""
import numpy as np
import pytest

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu

SIZES = (22_000, 180_000, 19_000, 18_000, 30_000, 21_000, 80_000, 15_000, 158_000, 141_000,
         11_000, 55_000)


def joined_states(scns):
    """The members' arrays back to back in page-locked memory, one array per field."""
    import torch
    sizes = [s.lc + 1 for s in scns]
    states, keep = [dict() for _ in scns], []
    for k, v in scns[0].state.items():
        if not isinstance(v, np.ndarray):
            for s, st in zip(scns, states):
                st[k] = s.state[k]
            continue
        t = torch.empty(sum(sizes), dtype=torch.from_numpy(v).dtype, pin_memory=True)
        keep.append(t)
        o = 0
        for s, st, n in zip(scns, states, sizes):
            st[k] = t.numpy()[o:o + n]
            st[k][:] = s.state[k]
            o += n
    return states, keep


def test_overlapping_chunks_of_mixed_element_sizes():
    scns = [S.config3_member(k, n, seed=3) for k, n in enumerate(SIZES)]
    prm = [X.make_params(s.params, n=1, tn=s.tn(1)) for s in scns]
    ref = [s.copy_state() for s in scns]
    bs = X.BatchSolver([s.grid for s in scns])
    bs.upload(ref)
    assert all(r.status == X.OK for r in bs.step_device(prm))
    bs.download(ref)
    bs.close()
    for _ in range(3):  # fresh contexts: the first call of each is the one that overlaps most
        states, _keep = joined_states(scns)
        bs = X.BatchSolver([s.grid for s in scns])
        assert all(r.status == X.OK for r in bs.step(prm, states))
        bs.close()
        for m, (a, b) in enumerate(zip(states, ref)):
            for k in ("p", "hp", "hu", "hv", "uhdye", "vhdxe", "uhe", "vhe", "lopenbcdry"):
                assert np.array_equal(a[k][1:scns[m].la], b[k][1:scns[m].la]), (m, k)
