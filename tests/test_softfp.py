"""softfp.cuh: the integer division, reciprocal, square root and multiplication
of the FP64 kernels give the bits of the IEEE operations (the host's), for every shape of
significand, next to exact quotients and squares, for special values, and with
the hardware estimates moved to either side of their error bound."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("softfp") / "harness")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "softfp_harness.cpp"), "-o", exe],
                   check=True)
    return exe


@pytest.mark.parametrize("error", [-2, 0, 2])
@pytest.mark.parametrize("pattern", range(8))
def test_bits_of_ieee(harness, pattern, error):
    out = subprocess.run([harness, str(pattern), "300000", str(error)], check=True, capture_output=True, text=True)
    assert out.stdout.strip() == "0"
