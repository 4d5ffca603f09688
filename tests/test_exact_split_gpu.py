"""The exact fractional form's split of few queries over segments: bit for bit the values of a call large enough to run
one query per thread, and the oracle's, at the edges of warps, units and passes."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


def loop_boundary(n_seg, rng, dtype):
    """A closed loop of n_seg segments with uneven weights."""
    t = np.sort(rng.uniform(0, 2 * np.pi, n_seg))
    p = np.stack([np.cos(t), np.sin(t), 0.3 * np.sin(3 * t)], 1)
    w = rng.choice([1.0, 2.0, 0.5], size=(n_seg, 1))
    return np.concatenate([p, np.roll(p, -1, 0), w], 1).astype(dtype)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,n_seg", [(1, 1), (31, 3), (32, 4), (33, 5), (257, 24), (5_000, 130), (38_900, 500)])
def test_split_equals_unsplit_and_oracle(n, n_seg, dtype):
    import antipodal_gb300 as ag
    from oracle.oracle import Oracle
    rng = np.random.default_rng(n)
    bnd, x0 = loop_boundary(n_seg, rng, dtype), synth.random_unit(rng).astype(dtype)
    many = rng.uniform(-1.5, 1.5, size=(60_000, 3)).astype(dtype)
    q = np.ascontiguousarray(many[:n])
    with ag.CudaDispatcher() as disp:
        large, out = np.empty(len(many), dtype), np.empty(n, dtype)
        ag.eval_gwnr_mesh_batch_fractional(disp, many, large, x0, bnd)
        for _ in range(2):  # the counters are left zeroed
            out[:] = 0
            ag.eval_gwnr_mesh_batch_fractional(disp, q, out, x0, bnd)
            assert np.array_equal(out, large[:n])
    few = slice(0, min(n, 200))
    ref = Oracle().frac_batch(q[few], x0, bnd)
    assert np.max(np.abs(out[few] - ref)) <= (1e-12 if dtype is np.float64 else 2e-5)
