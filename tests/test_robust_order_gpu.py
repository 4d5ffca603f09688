"""The int64_grid evaluator keeps its boundary in chain order: shuffled boundaries at the edges of the ordering block
(1,024 entries) and of its limit (4,096 segments) give the oracle's values, in one launch per mesh and in a batch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def loops(n_seg, rng):
    """Closed loops of 3 to 40 segments around random centres (and what is left over as an open chain), shuffled."""
    rows = []
    while len(rows) < n_seg:
        m = min(int(rng.integers(3, 41)), n_seg - len(rows))
        t = np.sort(rng.uniform(0, 2 * np.pi, m + 1))
        p = rng.uniform(-1, 1, 3) + 0.2 * np.stack([np.cos(t), np.sin(t), 0.3 * np.sin(3 * t)], 1)
        if m > 2 and len(rows) + m < n_seg:
            p[-1] = p[0]
        rows += [np.concatenate([p[k], p[k + 1], [rng.choice([1.0, 2.0])]]) for k in range(m)]
    return np.array(rows)[rng.permutation(n_seg)]


@pytest.mark.parametrize("mode", ["exact", "mixed"])
@pytest.mark.parametrize("n_seg", [1, 2, 500, 978, 1023, 1024, 1025, 4096, 4097])
def test_shuffled_boundary(n_seg, mode):
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    from oracle.oracle import Oracle
    rng = np.random.default_rng(n_seg)
    bnd = loops(n_seg, rng)
    v, idx = rng.uniform(-1.2, 1.2, (30, 3)), rng.permutation(30).astype(np.int32)
    q = rng.uniform(-1.5, 1.5, (45_003, 3))
    q[:20] = bnd[np.arange(20) % n_seg, 0:3]
    disp = ag.CudaDispatcher(stream=torch.cuda.current_stream())
    disp.set_robust_precision(mode)
    mesh = ag.CudaRobustMeshGwn(disp, v, idx, bnd, precision="int64_grid")
    p = torch.from_numpy(q).cuda()
    big, few = torch.empty(len(q), dtype=torch.float64, device="cuda"), torch.empty(300, dtype=torch.float64, device="cuda")
    mesh.evaluate(p, big)
    mesh.evaluate(p[:300].contiguous(), few)
    assert torch.equal(few, big[:300])
    out = torch.empty_like(big)
    ag.CudaRobustBatch(disp, [mesh], [p], [out]).run(graph=False)
    torch.cuda.synchronize()
    assert torch.equal(out, big)
    ref = Oracle().robust_eval("int64_grid", v, idx, bnd, q[:300])[0]
    # a sum of n_seg terms below pi in another order: some ulps of its partial sums; mixed: 6e-8 a term at most
    tol = 1e-12 + 1e-14 * n_seg if mode == "exact" else 6e-8 * n_seg / np.pi
    assert np.max(np.abs(few.cpu().numpy() - ref)) <= tol
