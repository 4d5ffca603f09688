"""The patch counts with the patches split over blocks (few queries): the counts and degenerate decisions of a call large
enough to run unsplit, and the added form equal to one sum, at the edges of groups and warps."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("patches", [1, 4, 5, 24, 150])
@pytest.mark.parametrize("n", [1, 33, 129, 3001])
def test_split_equals_unsplit(patches, n):
    import antipodal_gb300 as ag
    rng = np.random.default_rng(patches * 7 + n)
    p = rng.standard_normal((patches, 4, 4, 3))
    many = rng.uniform(-2.0, 2.0, size=(140_000, 3))
    many[: min(n, patches)] = p[: min(n, patches), 0, 0]  # on corners: degenerate decisions
    q = np.ascontiguousarray(many[:n])
    x0 = synth.random_unit(rng)
    with ag.CudaDispatcher() as d:
        isect = ag.CudaBezierPatchIntersector(d, p)
        got = [np.empty(n, np.int32) for _ in range(2)]
        want = [np.empty(len(many), np.int32) for _ in range(2)]
        ag.eval_gwnr_parametric_batch_integer(d, isect, many, want[0], x0, want[1])
        ag.eval_gwnr_parametric_batch_integer(d, isect, q, got[0], x0, got[1])
        frac = rng.standard_normal(n)
        added = frac.copy()
        assert ag.library().agwn_param_add_integer_bezier3x3_f64(d.handle, isect.handle, q.ctypes.data, n,
                                                                 added.ctypes.data, x0.ctypes.data) == 0
        isect.close()
    for a, b in zip(got, want):
        assert np.array_equal(a, b[:n])
    assert np.array_equal(added, frac + got[0])
