"""A batch's work list at the edges of its units (128, 256 and 512 queries): every configuration gives the one-mesh
evaluator's bits."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["mixed", "exact"])
@pytest.mark.parametrize("counts", [(1,), (127, 128, 129), (255, 0, 257), (511, 513), (1, 3, 1025)])
def test_item_units(gwn, mode, counts):
    torch = pytest.importorskip("torch")
    disp = gwn.CudaDispatcher(stream=torch.cuda.current_stream())
    disp.set_robust_precision(mode)
    rng = np.random.default_rng(sum(counts))
    v, i = synth.noisy_mesh("torus", 700, 5, rng)
    bnd = synth.boundary_segments(v, i)
    mesh = gwn.CudaRobustMeshGwn(disp, v, i, bnd, precision="int64_grid")
    pos = [torch.from_numpy(rng.uniform(v.min(0) * 1.2, v.max(0) * 1.2, (n, 3))).cuda() for n in counts]
    ref_out = [torch.empty(n, dtype=torch.float64, device="cuda") for n in counts]
    ref_cnt = [torch.empty(n, dtype=torch.int32, device="cuda") for n in counts]
    for p, o, c in zip(pos, ref_out, ref_cnt):
        if len(p):
            mesh.evaluate(p, o, c)
    out = [torch.empty_like(o) for o in ref_out]
    cnt = [torch.empty_like(c) for c in ref_cnt]
    batch = gwn.CudaRobustBatch(disp, [mesh] * len(counts), pos, out, cnt)
    for cfg in (None, (128, 1, 512, 64), (128, 2, 64, 64), (256, 1, 512, 64), (256, 2, 32, 64)):
        if cfg:
            batch.set_config(*cfg)
        for graph in (False, True):
            for o, c in zip(out, cnt):
                o.fill_(float("nan"))
                c.fill_(-7)
            batch.run(graph=graph)
            torch.cuda.synchronize()
            for a, b in zip(out + cnt, ref_out + ref_cnt):
                assert torch.equal(a, b), (cfg, graph)
