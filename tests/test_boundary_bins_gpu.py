"""Boundary extraction where its binning by lower vertex can go wrong: bins at and above the length that takes the radix
sort, repeated and degenerate edges, a vertex array far larger than the mesh, few rows of room.  The oracle's rows."""

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


def fan(k):
    """k triangles around vertex 0: its bin holds 2 k edges."""
    v = np.concatenate([np.zeros((1, 3)), np.random.default_rng(k).normal(size=(k + 1, 3))])
    i = np.stack([np.zeros(k, int), np.arange(1, k + 1), np.arange(2, k + 2)], 1)
    return v, i.astype(np.int32).ravel()




@pytest.mark.parametrize("k", [1, 255, 256, 257, 3000])
def test_fans(k):
    import antipodal_gb300 as ag
    v, i = fan(k)
    with ag.CudaDispatcher() as d:
        got = ag.build_boundary_segments(d, v, i)
    assert np.array_equal(got, synth.boundary_segments(v, i))


@pytest.mark.parametrize("kind", ["repeated", "degenerate", "sparse", "shuffled"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_odd_meshes(kind, dtype):
    import antipodal_gb300 as ag
    rng = np.random.default_rng(3)
    v, f = synth.noisy_mesh("torus", 3000, 5, rng)
    f = f.reshape(-1, 3)
    if kind == "repeated":
        f = np.concatenate([f, f[::3], f[::3], f[1::5][:, [0, 2, 1]]])
    elif kind == "degenerate":
        f[::7, 1] = f[::7, 0]
    elif kind == "sparse":
        big = np.zeros((1_000_000, 3))
        big[::300][: len(v)] = v
        v, f = big, f * 300
    else:
        f = f[rng.permutation(len(f))]
    v, i = v.astype(dtype), np.ascontiguousarray(f.astype(np.int32)).ravel()
    want = synth.boundary_segments(v, i)
    with ag.CudaDispatcher() as d:
        assert np.array_equal(ag.build_boundary_segments(d, v, i), want)
        fn = getattr(ag.library(), "agwn_build_boundary_segments_" + ("f64" if dtype is np.float64 else "f32"))
        import ctypes
        n, some = ctypes.c_int64(), np.zeros((5, 7), dtype)
        assert fn(d.handle, v.ctypes.data, len(v), i.ctypes.data, len(i), some.ctypes.data, 5, ctypes.byref(n)) == 0
    assert n.value == len(want) and np.array_equal(some, want[:5])
