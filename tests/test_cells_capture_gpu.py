"""A call captured into a CUDA graph after one warm-up keeps the cell grid it was captured with: later calls on the mesh,
which would otherwise build a finer one, leave the graph's results and their own as they were."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n", [("exact", 500), ("exact", 50_000), ("mixed", 50_000)])
def test_capture_after_one_call(precision, n):
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    v, idx, b, _, x0 = synth.open_icosphere(0, 4, grid=2)
    rng = np.random.default_rng(n)
    p = torch.from_numpy(rng.uniform(-1.3, 1.3, (n, 3))).cuda()
    bnd = torch.from_numpy(b).cuda()
    out, direct = torch.empty(n, dtype=torch.float64, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        disp = ag.CudaDispatcher(stream=s)
        disp.set_precision(precision)
        mesh = ag.CudaIntersector(disp, v, idx)
        ag.eval_gwnr_mesh_batch(disp, mesh, p, out, x0, bnd)
        s.synchronize()
        want = out.clone()
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            ag.eval_gwnr_mesh_batch(disp, mesh, p, out, x0, bnd)
        for _ in range(3):
            ag.eval_gwnr_mesh_batch(disp, mesh, p, direct, x0, bnd)
            s.synchronize()
            assert torch.equal(direct, want)
            out.fill_(float("nan"))
            graph.replay()
            s.synchronize()
            assert torch.equal(out, want)
        disp.synchronize()
