"""The double-float operators of the mixed parametric form (csrc/df32.cuh) on the host build of the same source: no mean or
largest error over random operands above that of the plain operators (tests/cpp/df32_check.cc)."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = str(tmp_path_factory.mktemp("df32") / "df32_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "df32_check.cc")], check=True)
    rows = subprocess.run([exe], stdout=subprocess.PIPE, check=True, text=True).stdout.splitlines()
    return {r.split()[0]: [float(x) for x in r.split()[1:]] for r in rows}


@pytest.mark.parametrize("name", ["quotient", "root", "fma", "dot", "det"])
def test_errors_no_larger_than_plain(errors, name):
    mean, most, plain_mean, plain_most = errors[name]
    # (the root's residual is formed in another order: equal to a percent)
    slack = 1.01 if name == "root" else 1.0
    assert mean <= plain_mean * slack and most <= plain_most * slack, errors[name]
