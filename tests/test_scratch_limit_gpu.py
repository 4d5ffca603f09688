"""Calls whose intermediate results exceed the scratch that there is (here: the context's limit) take them in smaller
pieces, with the same bits: the parametric integrals by queries and by curves, the split exact forms' terms by segments."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


def limited(ag, limit):
    from antipodal_gb300 import _lib
    d = ag.CudaDispatcher()
    d.set_option(_lib.OPT_SCRATCH_LIMIT, limit)
    assert d.get_option(_lib.OPT_SCRATCH_LIMIT) == limit
    return d


def device(a):
    torch = pytest.importorskip("torch")
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    torch.cuda.synchronize()
    return t


# 201 queries x 48 curves: pieces of queries that divide neither, one query at a time, and (exact) pieces of its curves
@pytest.mark.parametrize("precision,limits", [("exact", (40_000, 1_000, 100)), ("mixed", (40_000, 4_700))])
@pytest.mark.parametrize("scale", [1.0, 1.3])
def test_parametric_integrals(precision, limits, scale):
    import antipodal_gb300 as ag
    curves, q, x0 = synth.bezier_patches(seed=2, n_patches=12, n_queries=201, near_dist=1e-1)
    x0 = x0 * scale
    p, c = device(q), device(curves)
    cfg = ag.IntegrateConfig(tol=1e-7)
    out = {}
    for limit in (0,) + limits:
        with limited(ag, limit) as d:
            d.set_param_precision(precision)
            o = device(np.full(len(q), np.nan))
            ag.eval_gwnr_parametric_batch_fractional(d, p, o, x0, c, cfg)
            d.synchronize()
            out[limit] = o.cpu().numpy()
    for limit in limits:
        np.testing.assert_array_equal(out[limit], out[0])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("limit", [200_000, 30_000, 2_500])
def test_mesh_terms(dtype, limit):
    import antipodal_gb300 as ag
    rng = np.random.default_rng(5)
    bnd = np.concatenate([rng.uniform(-1, 1, (307, 6)), rng.integers(1, 3, (307, 1))], 1).astype(dtype)
    q = rng.uniform(-1.5, 1.5, (300, 3)).astype(dtype)
    x0 = np.array([0.36, 0.48, 0.8], dtype)
    p, b = device(q), device(bnd)
    out = []
    for lim in (0, limit):
        with limited(ag, lim) as d:
            o = device(np.full(len(q), np.nan, dtype))
            ag.eval_gwnr_mesh_batch_fractional(d, p, o, x0, b)
            d.synchronize()
            out.append(o.cpu().numpy())
    np.testing.assert_array_equal(out[1], out[0])


@pytest.mark.parametrize("policy,dtype", [("int64_grid", np.float32), ("int64_grid", np.float64),
                                          ("int128_grid", np.float64), ("exact_float", np.float64)])
@pytest.mark.parametrize("limit", [200_000, 30_000, 5_000])
def test_robust_terms(policy, dtype, limit):
    import antipodal_gb300 as ag
    from antipodal_gb300 import _lib
    v, idx, bnd, q = synth.two_tori(seed=1, n_tris=4_000, n_holes=5, n_queries=300, dtype=dtype)
    p = device(q)
    with ag.CudaDispatcher() as d:
        mesh = ag.CudaRobustMeshGwn(d, v, idx, bnd, precision=policy)
        out = []
        for lim in (0, limit):
            d.set_option(_lib.OPT_SCRATCH_LIMIT, lim)
            o, f = (device(np.full(len(q), np.nan, dtype)) for _ in range(2))
            counts = device(np.zeros(len(q), np.int32))
            mesh.evaluate(p, o, counts, f)
            d.synchronize()
            out.append((o.cpu().numpy(), counts.cpu().numpy(), f.cpu().numpy()))
        for a, b in zip(*out):
            np.testing.assert_array_equal(b, a)
        mesh.close()


def test_calls_that_cannot_be_cut():
    import antipodal_gb300 as ag
    with limited(ag, 1_000) as d:
        with pytest.raises(ag.GwnError) as e:
            ag.eval_gwnr_mesh_batch_fractional(d, np.zeros((500, 3)), np.empty(500), np.array([0.0, 0.0, 1.0]),
                                               np.ones((1, 7)))
        assert e.value.status == 3


def test_boundary_fallback_takes_the_sort_alone():
    """A vertex array far larger than its triangles use takes the radix sort (36 bytes per edge and its counters), without
    the 16 bytes per edge of the bins."""
    import antipodal_gb300 as ag
    n_tri = 20_000
    rng = np.random.default_rng(1)
    v = rng.normal(size=(16 * 3 * n_tri + 70_000, 3))
    idx = rng.integers(0, len(v), 3 * n_tri).astype(np.int32)
    with ag.CudaDispatcher() as d:
        want = ag.build_boundary_segments(d, v, idx)
    vt, it = device(v), device(idx)
    with limited(ag, 2_900_000) as d:
        got = ag.build_boundary_segments(d, vt, it).cpu().numpy()
    np.testing.assert_array_equal(got, want)
