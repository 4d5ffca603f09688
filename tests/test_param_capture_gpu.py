"""The exact parametric integrator's table of node bases is filled by the first call.  When that call is captured into a
graph (a relaxed capture, which may allocate), the table is filled only when the graph runs: a direct call before then has
to fill it for itself."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


def test_first_exact_call_captured():
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    curves, q, x0 = synth.bezier_patches(seed=4, n_patches=2, n_queries=40, near_dist=1e-1)
    cfg = ag.IntegrateConfig(tol=1e-8)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        p, c = torch.from_numpy(q).cuda(), torch.from_numpy(curves).cuda()
        out, direct = (torch.full((len(q),), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
        disp = ag.CudaDispatcher(stream=s)
        disp.set_param_precision("mixed")  # allocates the scratch that the exact form needs too
        ag.eval_gwnr_parametric_batch_fractional(disp, p, out, x0, c, cfg)
        s.synchronize()
        disp.set_param_precision("exact")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s, capture_error_mode="relaxed"):
            ag.eval_gwnr_parametric_batch_fractional(disp, p, out, x0, c, cfg)
        ag.eval_gwnr_parametric_batch_fractional(disp, p, direct, x0, c, cfg)
        s.synchronize()
        graph.replay()
        s.synchronize()
        want = np.empty(len(q))
        with ag.CudaDispatcher() as fresh:
            ag.eval_gwnr_parametric_batch_fractional(fresh, q, want, x0, curves, cfg)
        np.testing.assert_array_equal(direct.cpu().numpy(), want)
        np.testing.assert_array_equal(out.cpu().numpy(), want)
        disp.close()
