"""The robust exact form's split of few queries over segments: bit for bit the values of a call large enough to run one
query per thread, under every policy, with near, grazing and far queries (differences beyond the short integer form)."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("policy,dtype", [("int64_grid", np.float32), ("int64_grid", np.float64),
                                          ("int128_grid", np.float64), ("exact_float", np.float64)])
@pytest.mark.parametrize("n", [1, 33, 700])
def test_split_equals_unsplit_and_oracle(policy, dtype, n):
    import antipodal_gb300 as ag
    from oracle.oracle import Oracle
    v, idx, bnd, many = synth.two_tori(seed=n, n_tris=2_000, n_holes=5, n_queries=50_000, dtype=dtype)
    few = np.ascontiguousarray(many[-n:])  # the last half lies 1e-9 to 1e-3 off the surface
    few[::3] = v[: len(few[::3])]          # on vertices
    few[1::3] *= 40                        # beyond 16 extents: differences above 2^24
    if n > 8:
        few[2::3] = bnd[np.arange(len(few[2::3])) % len(bnd), 0:3] + np.array([3, 0, 0], dtype)  # rays through vertices
    all_q = np.concatenate([few, many])
    with ag.CudaDispatcher() as disp:
        r = ag.CudaRobustMeshGwn(disp, v, idx, bnd, precision=policy)
        big = [np.empty(len(all_q), t) for t in (dtype, np.int32, dtype)]
        out = [np.empty(n, t) for t in (dtype, np.int32, dtype)]
        r.evaluate(all_q, *big)
        r.evaluate(few, *out)
        r.close()
    for a, b in zip(out, big):
        assert np.array_equal(a, b[:n])
    gw, counts, frac = Oracle().robust_eval(policy, v, idx, bnd, few)
    assert np.array_equal(out[1], counts)
    assert np.max(np.abs(out[2].astype(np.float64) - frac)) <= (1e-12 if dtype is np.float64 else 2e-7)
