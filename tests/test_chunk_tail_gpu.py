"""Calls that run in chunks on two streams and whose last chunk holds so few queries that the exact form shares them out by
segment: the values are those of the same queries in one piece."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("tail", [5, 3_001])
def test_short_last_chunk(dtype, host, tail):
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    v, idx, bnd, _, x0 = synth.rotated_open_cube(seed=4, n_queries=0, dtype=dtype)
    n = (2 << 20) + tail  # chunks of 2^20, 2^20 and the tail
    q = np.random.default_rng(tail).uniform(-1.5, 1.5, (n, 3)).astype(dtype)
    with ag.CudaDispatcher() as disp:
        isect = ag.CudaIntersector(disp, v, idx)
        want = np.empty(n, dtype)
        for a in range(0, n, 700_000):  # below every chunked size
            ag.eval_gwnr_mesh_batch(disp, isect, q[a:a + 700_000], want[a:a + 700_000], x0, bnd)
        for _ in range(3):
            if host:
                got = np.full(n, np.nan, dtype)
                ag.eval_gwnr_mesh_batch(disp, isect, q, got, x0, bnd)
            else:
                out = torch.full((n,), float("nan"), dtype=torch.from_numpy(want).dtype, device="cuda")
                p = torch.from_numpy(q).cuda()
                torch.cuda.synchronize()
                ag.eval_gwnr_mesh_batch(disp, isect, p, out, x0, bnd)
                disp.synchronize()
                got = out.cpu().numpy()
            np.testing.assert_array_equal(got, want)
        isect.close()
