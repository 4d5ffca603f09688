"""Contexts on several host threads share one robust evaluator: its first calls, which build the cell grid, may run at
the same time."""

import threading

import numpy as np
import pytest

from antipodal_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("policy,dtype", [("int64_grid", np.float32), ("exact_float", np.float64)])
def test_first_calls_at_the_same_time(policy, dtype):
    import antipodal_gb300 as ag
    v, idx, bnd, q = synth.two_tori(seed=3, n_tris=40_000, n_holes=3, n_queries=2_000, dtype=dtype)
    with ag.CudaDispatcher() as disp:
        alone = ag.CudaRobustMeshGwn(disp, v, idx, bnd, precision=policy)
        want = np.empty(len(q), np.int32)
        alone.evaluate(q, np.empty(len(q), dtype), want)
        alone.close()
        others = [ag.CudaDispatcher() for _ in range(2)]
        for _ in range(6):
            mesh = ag.CudaRobustMeshGwn(disp, v, idx, bnd, precision=policy)
            counts = [np.empty(len(q), np.int32) for _ in others]
            barrier, failed = threading.Barrier(len(others)), []

            def first(k):
                try:
                    barrier.wait()
                    mesh.evaluate(q, np.empty(len(q), dtype), counts[k], dispatcher=others[k])
                except Exception as e:  # noqa: BLE001 - reported by the test's thread
                    failed.append(e)

            threads = [threading.Thread(target=first, args=(k,)) for k in range(len(others))]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            assert not failed, failed
            for c in counts:
                np.testing.assert_array_equal(c, want)
            mesh.close()
        for d in others:
            d.close()
