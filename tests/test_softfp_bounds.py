"""softfp.cuh at the error bounds its digits are derived from: on the host with the
estimates moved to their bounds, on the GPU the hardware's estimates over all
arguments and the device's branches against its IEEE operations."""
import ctypes
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
with open(os.path.join(HERE, "..", "geon_gb300", "csrc", "softfp.cuh")) as f:
    RCP_ERROR, RSQRT_ERROR = (float.fromhex(v) for v in re.search(
        r"RCP_ERROR = (0x[0-9.]+p-\d+), RSQRT_ERROR = (0x[0-9.]+p-\d+)", f.read()).groups())


def test_bounds_in_their_sums():
    # with the arguments' rounding: what the digits of the quotient and of the root are derived from
    assert RCP_ERROR + 2.0 ** -24 <= 2.0 ** -21.67 and RSQRT_ERROR + 2.0 ** -24 <= 2.0 ** -22


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("softfp") / "harness")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "softfp_bound_harness.cpp"), "-o", exe],
                   check=True)
    return exe


@pytest.mark.parametrize("part", ["-1", "-0.5", "0.5", "1"])
@pytest.mark.parametrize("pattern", range(8))
def test_bits_at_the_bounds(harness, pattern, part):
    out = subprocess.run([harness, str(pattern), "400000", part], check=True, capture_output=True, text=True)
    assert out.stdout.strip() == "0"


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    from geon_gb300 import build
    out = str(tmp_path_factory.mktemp("softfp") / "libdevice_harness.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "--fmad=false", "-shared",
                    os.path.join(HERE, "softfp_device_harness.cu"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.worst_estimate.restype = ctypes.c_double
    lib.wrong_operations.restype = ctypes.c_ulonglong
    lib.wrong_operations.argtypes = [ctypes.c_int, ctypes.c_ulonglong]
    return lib


@pytest.mark.gpu
def test_hardware_estimates_over_all_arguments(device):
    # the measured error is formed in FP64, off by a few 2^-53
    assert 0.0 < device.worst_estimate(0) <= RCP_ERROR - 2.0 ** -50
    assert 0.0 < device.worst_estimate(1) <= RSQRT_ERROR - 2.0 ** -45  # (without the e^2 / 2 of the square)


@pytest.mark.gpu
@pytest.mark.parametrize("pattern", range(8))
def test_device_bits_of_ieee(device, pattern):
    assert device.wrong_operations(pattern, 1 << 24) == 0
