"""The exact parametric form at the edges of its work split: fewer pairs than teams, one query, one curve, trees below
and above the tabulated depth.  Bit for bit the oracle's values."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,patches,drop", [(1, 1, 3), (1, 3, 0), (7, 1, 3), (33, 2, 1), (129, 3, 0)])
@pytest.mark.parametrize("max_depth", [0, 10, 13])
def test_teams_equal_oracle(n, patches, drop, max_depth):
    import antipodal_gb300 as ag
    from oracle.oracle import Oracle
    curves, q, x0 = synth.bezier_patches(seed=n, n_patches=patches, n_queries=n)
    curves = np.ascontiguousarray(curves[:len(curves) - drop])
    cfg = ag.IntegrateConfig(0, max_depth, 1e-12)
    with ag.CudaDispatcher() as disp:
        out, nodes = np.empty(n), np.empty(n, np.int32)
        ag.eval_gwnr_parametric_batch_fractional(disp, q, out, x0, curves, cfg, nodes_per_query=nodes)
    ref, _, _ = Oracle().param_frac_bezier3(q, x0, curves, 0, max_depth, 1e-12, stats=True)
    assert np.array_equal(out, ref)
    if max_depth == 0:
        assert (nodes == len(curves)).all()
