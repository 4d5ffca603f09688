"""A graph captured from a call on few queries keeps the scratch it was captured with: a later call with more queries, which
needs more, must not free it."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_larger_call_between_replays(dtype):
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    _, _, bnd, _, x0 = synth.open_icosphere(0, 3, grid=2)
    rng = np.random.default_rng(3)
    x0 = x0.astype(dtype)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        few, many = (torch.from_numpy(rng.uniform(-1.3, 1.3, (n, 3)).astype(dtype)).cuda() for n in (300, 30_000))
        b = torch.from_numpy(bnd.astype(dtype)).cuda()
        out, out_many = torch.empty_like(few[:, 0].contiguous()), torch.empty_like(many[:, 0].contiguous())
        disp = ag.CudaDispatcher(stream=s)
        ag.eval_gwnr_mesh_batch_fractional(disp, few, out, x0, b)
        s.synchronize()
        want = out.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            ag.eval_gwnr_mesh_batch_fractional(disp, few, out, x0, b)
        for _ in range(2):
            ag.eval_gwnr_mesh_batch_fractional(disp, many, out_many, x0, b)
            s.synchronize()
            filler = [torch.full((1 << 16,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(8)]
            out.fill_(0)
            graph.replay()
            s.synchronize()
            assert torch.equal(out, want)
            assert all(bool(torch.isnan(f).all()) for f in filler)
        del graph
        disp.trim()
        ag.eval_gwnr_mesh_batch_fractional(disp, few, out, x0, b)
        s.synchronize()
        assert torch.equal(out, want)
        disp.close()
