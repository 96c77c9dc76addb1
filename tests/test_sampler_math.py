"""The FP64 sampler functions (csrc/kpmath.cuh), compiled for the host, against 80-bit arithmetic."""
import os
import subprocess

import pytest

import _oracle as O


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("kpmath") / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(O.REPO, "masterarbeit_b200", "csrc"),
                    os.path.join(O.REPO, "tests", "kpmath_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {f[0]: (float(f[1]), float(f[2])) for f in (line.split() for line in out.splitlines())}


def test_quotient_by_beta(errors):
    # a correctly rounded division is off by 1/2 ulp at most, 1/sqrt(12) rms; the lo part leaves 2^-52 of that
    assert errors["over_beta"][0] <= 0.5001 and errors["over_beta"][1] <= 0.2895
    assert errors["limits"][0] == 1   # beta = inf, 0, below the normal range, negative
