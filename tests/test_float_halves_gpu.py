"""Float full calls run in two halves from 786,432 queries: at the edges of the rule, the fractional call's values plus the
integer call's, which run in one piece, bit for bit."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [786_431, 786_432, 786_433, 787_457, 2_097_151, 2_097_152])
def test_halves(n):
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    v, idx, b, _, x0 = synth.open_icosphere(1, 3, grid=2, dtype=np.float32)
    g = torch.Generator(device="cuda").manual_seed(n)
    p = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float32) * 2.4 - 1.2
    bnd = torch.from_numpy(b).cuda()
    full = torch.full((n,), float("nan"), dtype=torch.float32, device="cuda")
    frac, cnt = torch.empty_like(full), torch.empty(n, dtype=torch.int32, device="cuda")
    disp = ag.CudaDispatcher(stream=torch.cuda.current_stream())
    mesh = ag.CudaIntersector(disp, v, idx)
    for _ in range(2):
        ag.eval_gwnr_mesh_batch(disp, mesh, p, full, x0, bnd)
    ag.eval_gwnr_mesh_batch_fractional(disp, p, frac, x0, bnd)
    ag.eval_gwnr_mesh_batch_integer(disp, mesh, p, cnt, x0)
    torch.cuda.synchronize()
    assert torch.equal(full, frac + cnt)
