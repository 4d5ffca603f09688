"""The exact form in float, with one query per thread or packed pairs: the same bits for every setting and for the split of
few queries, zeros, infinities and NaN handled as the reference's float arithmetic handles them."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e12, 1e-22, 1e19])
@pytest.mark.parametrize("n", [40_001, 65_537])
def test_same_bits_and_oracle(n, scale):
    import antipodal_gb300 as ag
    from oracle.oracle import Oracle
    rng = np.random.default_rng(n)
    p = rng.uniform(-1, 1, (34, 3))
    w = rng.choice([1.0, 2.0, 0.5], (33, 1))
    bnd = (np.concatenate([p[:-1], p[1:], w], 1) * np.r_[np.full(6, scale), 1.0]).astype(np.float32)
    x0 = synth.random_unit(rng).astype(np.float32)
    q = (rng.uniform(-1.5, 1.5, (n, 3)) * scale).astype(np.float32)
    q[0:33] = bnd[:, 0:3]                       # on vertices
    q[33:66] = 0.5 * (bnd[:, 0:3] + bnd[:, 3:6])  # on segments
    q[66], q[67, 1], q[68, 2] = 0, np.inf, np.nan
    outs = []
    for k in (1, 2, 4, 8):
        with ag.CudaDispatcher(queries_per_thread=k) as disp:
            out, few = np.empty(n, np.float32), np.empty(101, np.float32)
            ag.eval_gwnr_mesh_batch_fractional(disp, q, out, x0, bnd)
            ag.eval_gwnr_mesh_batch_fractional(disp, np.ascontiguousarray(q[:101]), few, x0, bnd)
        outs += [out, few]
    for a in outs[1:]:
        assert np.array_equal(a, outs[0][:len(a)], equal_nan=True)
    assert np.isnan(outs[0][68])
    ref = Oracle().frac_batch(q[66:500], x0, bnd)
    good = np.isfinite(ref)
    assert np.array_equal(np.isnan(ref), np.isnan(outs[0][66:500]))
    # 33 terms of at most pi w; both sides evaluate the same float products and sums and differ in atan2 alone, by some
    # ulps of a term (4 ulp of pi: 1e-6), in the weights' sum of 33 x 2
    assert np.max(np.abs(outs[0][66:500][good] - ref[good])) <= 66 * 1e-6 / (2 * np.pi)
