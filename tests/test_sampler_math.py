"""The FP64 sampler functions (csrc/kpmath.cuh), compiled for the host, against 80-bit arithmetic."""
import os
import subprocess
import sys

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


@pytest.mark.parametrize("name,largest,rms", [("log", 0.54, 0.29), ("cos2", 3.38, 0.784), ("sin", 1.48, 0.36), ("cos", 1.48, 0.36)])
def test_functions_of_a_word(errors, name, largest, rms):
    # no worse than the CUDA library functions in their place: errors measured on the device over 12 million words
    assert errors[name][0] <= largest and errors[name][1] <= rms


def test_the_header_holds_the_generated_constants():
    pytest.importorskip("mpmath")
    sys.path.insert(0, os.path.join(O.REPO, "tests", "golden"))
    import make_kpmath

    text = open(os.path.join(O.REPO, "masterarbeit_b200", "csrc", "kpmath.cuh")).read()
    for block in make_kpmath.blocks():
        assert block in text, block.split("\n")[0]
