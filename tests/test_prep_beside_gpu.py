"""A mixed full call prepares its boundary on a second stream beside the counts: alternating boundaries, meshes and sizes
without a wait in between give the fractional call's values plus the integer call's, bit for bit."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(700, 5_001, 90_000), (200_003, 900, 30_000)])
def test_full_is_fraction_plus_counts(sizes):
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    rng = np.random.default_rng(sum(sizes))
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        disp = ag.CudaDispatcher(stream=s)
        disp.set_precision("mixed")
        work = []
        for n, level in zip(sizes, (4, 6, 5)):
            v, idx, b, _, x0 = synth.open_icosphere(n, level, grid=2)
            p = torch.from_numpy(rng.uniform(-1.3, 1.3, (n, 3))).cuda()
            mesh, bnd = ag.CudaIntersector(disp, v, idx), torch.from_numpy(b).cuda()
            frac = torch.empty(n, dtype=torch.float64, device="cuda")
            cnt = torch.empty(n, dtype=torch.int32, device="cuda")
            ag.eval_gwnr_mesh_batch_fractional(disp, p, frac, x0, bnd)
            ag.eval_gwnr_mesh_batch_integer(disp, mesh, p, cnt, x0)
            work.append((mesh, p, x0, bnd, frac + cnt))
        outs = [[torch.full_like(w[4], float("nan")) for w in work] for _ in range(4)]
        for rep in outs:
            for (mesh, p, x0, bnd, _), out in zip(work, rep):
                # the boundary is a copy that lives no longer than the call
                ag.eval_gwnr_mesh_batch(disp, mesh, p, out, x0, bnd.clone())
        s.synchronize()
    for rep in outs:
        for w, out in zip(work, rep):
            assert torch.equal(out, w[4])
