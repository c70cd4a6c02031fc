"""A context's first transfers of pageable arrays allocate nothing: what they go through
is there since its creation (page-locking and allocating it took the first call several
milliseconds)."""
import pytest
import torch

import efdc_xm as X
import scenario as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(140, 133), (250, 200), (600, 500)])
def test_no_allocation(nx, ny):
    torch.zeros(1, device="cuda")
    scn = S.make_scenario(nx, ny, seed=3, depth=(4.0, 30.0), amp=0.4, fill_dead_ends=True)
    warm = X.Solver(scn.grid)  # (modules and streams of the process)
    st = scn.copy_state()
    warm.upload(st)
    warm.download(st)
    sol = X.Solver(scn.grid)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    sol.download(st)
    sol.upload(st)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    sol.close()
    warm.close()
