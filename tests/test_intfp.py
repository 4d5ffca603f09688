"""The exact forms' division, square root, product and atan2 on the integer pipe (csrc/intfp.cuh): bit for bit IEEE
division, square root and product, and atan2 within 3 ulp, on the host build of the same source (CPU) and on the device."""

import os
import re
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = os.path.join(ROOT, "antipodal_gb300", "csrc", "intfp.cuh")


def pairs(kind: str, n: int = 40_000):
    rng = np.random.default_rng(11)
    bits = rng.integers(0, 1 << 64, size=(2, n), dtype=np.uint64)
    if kind == "any bits":  # every exponent, infinities, NaN and subnormals among them
        return bits.view(np.float64)
    if kind == "specials":
        v = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308,
                      1.7976931348623157e308, 4.450147717014403e-308, 8.98846567431158e307, 3.0, 1 / 3, 2.0 ** 383,
                      2.0 ** 384, 2.0 ** -383, 2.0 ** -384])
        a, b = np.meshgrid(v, v)
        return np.stack([a.ravel(), b.ravel()])
    one = (bits & np.uint64((1 << 52) - 1)) | np.uint64(0x3FF << 52)
    if kind == "near one":  # quotients and roots next to 1, few or many trailing ones and zeros
        a = one[0] >> rng.integers(0, 52, n).astype(np.uint64) << rng.integers(0, 20, n).astype(np.uint64)
        a = (a & np.uint64((1 << 52) - 1)) | np.uint64(0x3FF << 52)
        b = a + rng.integers(0, 64, n).astype(np.uint64) - np.uint64(32)
        return np.stack([a, b]).view(np.float64)
    if kind == "halfway":  # quotients and roots as close to a halfway point as doubles come
        t = [int(x) >> 1 | 1 << 52 for x in one[0] & np.uint64((1 << 53) - 1)]
        d = [int(x) | 1 << 52 for x in one[1] & np.uint64((1 << 52) - 1)]
        a, b = [], []
        for k, (x, y) in enumerate(zip(t, d)):
            m = (2 * x + 1) * y if k % 2 else x * x + x
            s = max(0, m.bit_length() - 53)
            s += (s & 1) if k % 2 == 0 else 0
            a.append(float(((m >> s) + k % 3 - 1)) * 2.0 ** s)
            b.append(float(y))
        return np.array([a, b])
    if kind == "short":  # few significant bits: exact products, ties, and products next to ties
        a = rng.integers(1, 1 << 27, n) * 2 + 1
        b = rng.integers(1, 1 << 27, n) * 2 + 1
        return np.stack([a * 2.0 ** rng.integers(-400, 400, n).astype(float), -b.astype(float)])
    angles = rng.uniform(-np.pi, np.pi, n)  # "angles": the circle, the multiples of 1/64 and 1/128 and tiny ratios
    y, x = np.sin(angles), np.cos(angles)
    k = rng.integers(0, 129, n) / 128.0
    y[::3] = x[::3] * k[::3]
    y[1::3] *= 2.0 ** -rng.integers(0, 70, len(y[1::3])).astype(float)
    return np.stack([y, x]) * 2.0 ** rng.integers(-300, 300, n).astype(float)


KINDS = ["any bits", "specials", "near one", "halfway", "short", "angles"]


def check(a, b, quotient, root, angle, product):
    with np.errstate(all="ignore"):
        want_q, want_r = a / b, np.sqrt(a)
        same = lambda u, v: (u.view(np.uint64) == v.view(np.uint64)) | (np.isnan(u) & np.isnan(v))  # noqa: E731
        assert same(quotient, want_q).all(), (a[~same(quotient, want_q)][:3], b[~same(quotient, want_q)][:3])
        assert same(root, want_r).all(), a[~same(root, want_r)][:3]
        assert same(product, a * b).all(), (a[~same(product, a * b)][:3], b[~same(product, a * b)][:3])
        want = np.arctan2(a.astype(np.longdouble), b.astype(np.longdouble))
        assert (np.isnan(angle) == np.isnan(want)).all()
        ok = ~np.isnan(angle)
        assert (np.signbit(angle[ok]) == np.signbit(want[ok].astype(np.float64))).all()
        # (n - c d), (d + c n), their quotient and its atan are rounded once each, half an ulp of a term no larger
        # than the angle; the last sum adds half an ulp: 2.5
        ulp = np.spacing(np.abs(want[ok]).astype(np.float64)).astype(np.longdouble)
        assert (np.abs(angle[ok] - want[ok]) <= 3 * ulp).all()


@pytest.fixture(scope="module")
def host_build(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("intfp") / "intfp_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "intfp_check.cc")], check=True)
    return exe


@pytest.mark.parametrize("kind", KINDS)
def test_host_build(host_build, kind):
    a, b = pairs(kind)
    r = subprocess.run([host_build], input=np.ascontiguousarray(np.stack([a, b], 1)).tobytes(), stdout=subprocess.PIPE,
                       check=True)
    out = np.frombuffer(r.stdout, np.float64).reshape(-1, 4)
    check(a, b, *(np.ascontiguousarray(out[:, k]) for k in range(4)))


def test_table():
    """Every entry's angle is the nearest double to its c's, and within 2^-10 ulp of it."""
    mp = pytest.importorskip("mpmath")
    text = open(SOURCE).read()
    body = text[text.index("kAtanTable[260] = {"):]
    body = body[:body.index("};")]
    rows = [(float(c), float(v)) for c, v in re.findall(r"\{([^{},]+), ([^{},]+)\}", body)]
    assert len(rows) == 260
    with mp.workprec(160):
        for i, (c, angle) in enumerate(rows):
            t = mp.atan(mp.mpf(c))
            want = [t, mp.pi / 2 - t, mp.pi - t, mp.pi / 2 + t][i % 4]
            assert abs(c - (i // 4) / 64) <= 2.0 ** -20
            assert abs(want - mp.mpf(angle)) <= np.spacing(angle) * 2.0 ** -10


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_device(kind):
    import antipodal_gb300 as ag
    a, b = (np.ascontiguousarray(v) for v in pairs(kind))
    out = [np.empty_like(a) for _ in range(4)]
    with ag.CudaDispatcher() as disp:
        assert ag.library().agwn_probe_math_f64(disp.handle, a.ctypes.data, b.ctypes.data, len(a),
                                                *(o.ctypes.data for o in out)) == 0
    check(a, b, *out)
