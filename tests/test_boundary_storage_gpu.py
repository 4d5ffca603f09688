"""A boundary from build_boundary_segments owns its rows and no more, whatever room the extraction took."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("triangles", [0, 10, 9_000])  # none, the open cube's four segments, more than the first rows
def test_owned_rows(dtype, triangles):
    torch = pytest.importorskip("torch")
    import antipodal_gb300 as ag
    if triangles <= 10:
        v, idx = synth.CUBE_VERTS.astype(dtype), synth.CUBE_IDX_OPEN_Y[:3 * triangles]
    else:  # a soup: every edge is open
        v = np.random.default_rng(2).normal(size=(3 * triangles, 3)).astype(dtype)
        idx = np.arange(3 * triangles, dtype=np.int32)
    with ag.CudaDispatcher() as d:
        host = ag.build_boundary_segments(d, v, idx)
        dev = ag.build_boundary_segments(d, torch.from_numpy(v).cuda(), torch.from_numpy(idx).cuda())
    assert host.base is None and host.flags.owndata
    assert host.shape == ({0: 0, 10: 4, 9_000: 27_000}[triangles], 7)
    assert dev.untyped_storage().nbytes() == host.nbytes
    np.testing.assert_array_equal(dev.cpu().numpy(), host)
