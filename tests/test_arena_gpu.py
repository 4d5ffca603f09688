"""Build temporaries of a context: builds of alternating kinds and sizes share them (several chunks that become one, scopes
inside scopes), and what exceeds 1 GB is given back."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


def test_alternating_builds_equal_separate_contexts():
    import antipodal_gb300 as ag
    rng = np.random.default_rng(2)
    x0 = np.array([0.36, 0.48, 0.8])
    meshes = [synth.noisy_mesh(kind, n, holes, rng) for kind, n, holes in
              (("torus", 500, 1), ("icosphere", 60_000, 3), ("torus", 2_000, 2), ("icosphere", 200_000, 5), ("torus", 900, 1))]
    q = rng.uniform(-1.4, 1.4, (3_000, 3))

    def evaluate(disp, v, idx):
        bnd = ag.build_boundary_segments(disp, v, idx)
        isect = ag.CudaIntersector(disp, v, idx)
        out = [bnd]
        for robust in (None, "int64_grid", "exact_float"):
            o, c = np.empty(len(q)), np.empty(len(q), np.int32)
            if robust is None:
                ag.eval_gwnr_mesh_batch(disp, isect, q, o, x0, bnd)
                ag.eval_gwnr_mesh_batch_integer(disp, isect, q, c, x0)
            else:
                mesh = ag.CudaRobustMeshGwn(disp, v, idx, bnd, precision=robust)
                mesh.evaluate(q, o, c)
                mesh.close()
            out += [o, c]
        isect.close()
        return out

    with ag.CudaDispatcher() as shared:
        for v, idx in meshes + meshes[::-1]:
            got = evaluate(shared, v, idx)
            with ag.CudaDispatcher() as own:
                want = evaluate(own, v, idx)
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)


def test_more_than_a_gigabyte_is_given_back():
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    n = 12_000_000  # a soup of small triangles: 1.4 GB of temporaries for its hierarchy
    g = torch.Generator(device="cuda").manual_seed(1)
    at = torch.rand(n, 1, 3, generator=g, device="cuda")
    v = (at + 1e-3 * torch.rand(n, 3, 3, generator=g, device="cuda")).reshape(-1, 3).contiguous()
    idx = torch.arange(3 * n, dtype=torch.int32, device="cuda")
    p, counts = torch.rand(1_000, 3, device="cuda"), torch.empty(1_000, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with ag.CudaDispatcher() as disp:
        isect = ag.CudaIntersector(disp, v, idx)
        ag.eval_gwnr_mesh_batch_integer(disp, isect, p, counts, np.array([0, 0, 1], np.float32))
        disp.synchronize()
        before = torch.cuda.mem_get_info()[0]
        disp.trim()
        assert torch.cuda.mem_get_info()[0] - before < 1 << 30
        isect.close()
    del at, v, idx
    torch.cuda.empty_cache()
