"""The exact forms' arctangent (atan2_int, csrc/intfp.cuh) stays within 1.51 ulp at every angle, small ones above all, on the
host build of the same source (CPU) and on the device.

With u = 2^-53: from n / d = 3/256 on, (n - c d), (d + c n), their quotient and the polynomial's last sum err by u relative
each, 4 u |q| in all.  Below 1/64 |q| <= 1/256, and from there to 3/128 |q| <= 1/128: at most one ulp of the angle; higher up
less.  The last sum adds half an ulp and the table 2^-10.  Below 3/256 the quotient and the last sum are all there is."""

import subprocess

import numpy as np
import pytest

from test_intfp import host_build  # noqa: F401 - the fixture

KINDS = {"circle": 0, "up to 3/64": 1, "1/256 to 1/64": 2, "1/128 to 3/64": 3, "ratios of any size": 4, "next to 3/256": 5}


def arguments(kind, n=200_000):
    rng = np.random.default_rng(KINDS[kind])
    x = rng.uniform(1.0, 2.0, n)
    if kind == "circle":
        a = rng.uniform(-np.pi, np.pi, n)
        return np.sin(a), np.cos(a)
    if kind == "ratios of any size":
        return 2.0 ** rng.uniform(-60.0, 60.0, n), rng.choice([-1.0, 1.0], n) * x
    lo, hi = {"up to 3/64": (0.0, 3 / 64), "1/256 to 1/64": (1 / 256, 1 / 64), "1/128 to 3/64": (1 / 128, 3 / 64),
              "next to 3/256": (3 / 256 - 1e-6, 3 / 256 + 1e-6)}[kind]
    return x * rng.uniform(lo, hi, n), x


def check(kind, y, x, angle):
    want = np.arctan2(y.astype(np.longdouble), x.astype(np.longdouble))
    ulp = np.spacing(np.abs(want).astype(np.float64)).astype(np.longdouble)
    assert float(np.max(np.abs(angle - want) / ulp)) <= 1.51


@pytest.mark.parametrize("kind", KINDS)
def test_host_build(host_build, kind):  # noqa: F811
    y, x = arguments(kind)
    r = subprocess.run([host_build], input=np.ascontiguousarray(np.stack([y, x], 1)).tobytes(), stdout=subprocess.PIPE,
                       check=True)
    check(kind, y, x, np.frombuffer(r.stdout, np.float64).reshape(-1, 4)[:, 2])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_device(kind):
    import antipodal_gb300 as ag
    y, x = (np.ascontiguousarray(v) for v in arguments(kind))
    out = [np.empty_like(y) for _ in range(4)]
    with ag.CudaDispatcher() as disp:
        assert ag.library().agwn_probe_math_f64(disp.handle, y.ctypes.data, x.ctypes.data, len(y),
                                                *(o.ctypes.data for o in out)) == 0
    check(kind, y, x, out[2])
