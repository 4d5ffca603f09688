"""trim() gives a context's scratch and build temporaries back to the device; later calls take them anew."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


def test_trim_gives_memory_back():
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    v, idx, bnd, _, x0 = synth.open_icosphere(0, 7, grid=2)  # some 300,000 triangles
    q = np.random.default_rng(1).uniform(-1.2, 1.2, (300_000, 3))

    def run(disp, isect):
        out = np.empty(len(q))
        ag.eval_gwnr_mesh_batch(disp, isect, q, out, x0, bnd)
        return out

    with ag.CudaDispatcher(precision="mixed") as disp:
        isect = ag.CudaIntersector(disp, v, idx)
        want = run(disp, isect)
        # at least the hierarchy's temporaries (more than 100 bytes per triangle) and the queries and results
        kept = 100 * len(idx) // 3 + 32 * len(q)
        before = torch.cuda.mem_get_info()[0]
        disp.trim()
        assert torch.cuda.mem_get_info()[0] - before >= kept - (4 << 20)  # in the allocator's 2 MB pages
        np.testing.assert_array_equal(run(disp, isect), want)
        disp.trim()
        other = ag.CudaIntersector(disp, v, idx)  # a build after a trim
        np.testing.assert_array_equal(run(disp, other), want)
        isect.close()
        other.close()
