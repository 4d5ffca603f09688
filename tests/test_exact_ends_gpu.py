"""The exact fractional form on boundaries whose neighbouring segments share ends in every way, across staged tiles: bit
for bit the values of the split of few queries, which works every end out for itself, and the oracle's."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


def boundary(kind, n_seg, rng):
    p = rng.uniform(-1, 1, (n_seg + 1, 3))
    p[rng.uniform(size=p.shape) < 0.1] = 0.0
    a, b = p[:-1].copy(), p[1:].copy()
    if kind == "backward":      # P1 of each is P0 of the one before
        a, b = b, a
    elif kind == "mixed":       # forward, backward, P0 = P0 and P1 = P1 in any order
        turn = rng.uniform(size=n_seg) < 0.5
        a[turn], b[turn] = b[turn].copy(), a[turn].copy()
    elif kind == "zeros":       # equal vertices whose zeros differ in sign
        a[::2] = np.where(a[::2] == 0, -0.0, a[::2])
    elif kind == "repeated":    # the same segment again, and its reverse
        a[1::3], b[1::3] = a[0::3][:len(a[1::3])], b[0::3][:len(b[1::3])]
        a[2::3], b[2::3] = b[1::3][:len(a[2::3])], a[1::3][:len(b[2::3])]
    return np.concatenate([a, b, rng.choice([1.0, 2.0], size=(n_seg, 1))], 1)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["forward", "backward", "mixed", "zeros", "repeated"])
@pytest.mark.parametrize("n_seg,tile", [(1, 512), (2, 512), (67, 32)])
def test_shared_ends(kind, n_seg, tile, dtype):
    import antipodal_gb300 as ag
    from oracle.oracle import Oracle
    rng = np.random.default_rng(n_seg)
    bnd, x0 = boundary(kind, n_seg, rng).astype(dtype), synth.random_unit(rng).astype(dtype)
    q = rng.uniform(-1.5, 1.5, size=(45_001, 3)).astype(dtype)
    q[:50] = 0.0
    q[50:100, 1] = -0.0
    out, part = np.empty(len(q), dtype), np.empty(15_001, dtype)
    with ag.CudaDispatcher(seg_tile=tile) as disp:
        ag.eval_gwnr_mesh_batch_fractional(disp, q, out, x0, bnd)
        for s in range(0, len(q), 15_000):
            few = np.ascontiguousarray(q[s:s + 15_000])
            ag.eval_gwnr_mesh_batch_fractional(disp, few, part[:len(few)], x0, bnd)
            assert np.array_equal(part[:len(few)], out[s:s + len(few)], equal_nan=True), s
    ref = Oracle().frac_batch(q[100:300], x0, bnd)
    assert np.max(np.abs(out[100:300] - ref)) <= (1e-12 if dtype is np.float64 else 2e-5)
