"""The mixed kernel at the largest segment tiles: what does not fit an SM's shared memory runs in smaller tiles, and the
values are the same."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,qpt", [(1952, 8), (1984, 8), (2048, 8), (2048, 4)])
def test_largest_tiles(tile, qpt):
    import antipodal_gb300 as ag
    n_seg = 2_100  # two tiles of the largest size and more
    a = np.linspace(0, 2 * np.pi, n_seg, endpoint=False)
    p = np.stack([np.cos(a), np.sin(a), 0.2 * np.sin(5 * a)], 1)
    bnd = np.concatenate([p, np.roll(p, -1, 0), np.ones((n_seg, 1))], 1)
    q = np.random.default_rng(7).uniform(-1.3, 1.3, (5_003, 3))
    x0 = np.array([0.36, 0.48, 0.8])
    out = {}
    for t, k in ((512, 2), (tile, qpt)):
        with ag.CudaDispatcher(precision="mixed", mixed_min_pairs=0, seg_tile=t, queries_per_thread=k, block=256) as d:
            out[t] = np.empty(len(q))
            ag.eval_gwnr_mesh_batch_fractional(d, q, out[t], x0, bnd)
    np.testing.assert_array_equal(out[tile], out[512])
