"""Fast steps of the mixed path (planar steps under one combined test in the
orbit-plane frame, in renders without t, in sweeps and in the serving kernel, and
groups of flat Alcubierre steps) against the steps with the separate tests: the same
state after every group of 16 steps, the same classes and counts, bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from geon_gb300._util import dp

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ORBIT, RENDER, SWEEP, SERVE_CAMERA, SERVE_EQUATORIAL, CHART = range(6)


@pytest.fixture(scope="module")
def compare(geon, tmp_path_factory):
    from geon_gb300 import build
    out = str(tmp_path_factory.mktemp("planar") / "libplanar.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "--fmad=false", "-w", "-shared",
                    os.path.join(HERE, "planar_steps_harness.cu"), "-o", out, f"-L{build.OUT}", "-lgeon_gpu",
                    "-Xlinker", f"-rpath={build.OUT}"], check=True)
    f = ctypes.CDLL(out).compare_steps
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.c_double), ctypes.c_longlong, ctypes.c_double,
                  ctypes.c_longlong, ctypes.POINTER(ctypes.c_longlong)]

    def run(metric, config, y, step, cap):
        out = np.zeros((len(y), 4), dtype=np.int64)
        y = np.ascontiguousarray(y)
        assert f(metric.handle, config, dp(y), len(y), step, cap, out.ctypes.data_as(ctypes.POINTER(ctypes.c_longlong))) == 0
        return out
    return run


def null_states(metric, r, rng, inward):
    """Null rays from radii r in random directions of random planes."""
    n = len(r)
    y = np.zeros((n, 8))
    y[:, 0], y[:, 1] = rng.uniform(-3.0, 3.0, n), r
    y[:, 2], y[:, 3] = rng.uniform(0.3, 2.8, n), rng.uniform(-3.0, 3.0, n)
    a = np.where(inward, rng.uniform(0.0, np.pi / 2, n), rng.uniform(0.0, np.pi, n))
    psi = rng.uniform(0.0, 2.0 * np.pi, n)
    if metric == "schwarzschild":
        f = 1.0 - 2.0 / r
        y[:, 4], y[:, 5], area = 1.0 / np.sqrt(f), -np.cos(a) * np.sqrt(f), r
    else:
        y[:, 4], y[:, 5], area = 1.0, -np.cos(a) * np.sign(r), np.sqrt(1.0 + r * r)
    y[:, 6] = np.sin(a) * np.sin(psi) / area
    y[:, 7] = np.sin(a) * np.cos(psi) / (area * np.sin(y[:, 2]))
    return y


def on_equator(y):
    y = y.copy()
    y[:, 2] = np.pi / 2
    y[:, 7] = np.hypot(y[:, 6], y[:, 7])
    y[:, 6] = 0.0
    return y


def check(out, fast=0.5):
    assert np.all(out[:, 0] == 0), out[out[:, 0] != 0][:5]
    assert out[:, 3].sum() > fast * out[:, 2].sum()  # the fast steps did run


@pytest.mark.parametrize("config", [ORBIT, RENDER, SWEEP, SERVE_CAMERA, SERVE_EQUATORIAL])
@pytest.mark.parametrize("step,cap,pad,escape", [
    (0.05, 6000, 1.001, 60.0), (0.01, 1003, 1.001, 100.0), (0.5, 400, 1.001, 50.0), (-0.05, 905, 1.001, 60.0),
    (0.05, 3000, 1.8, 45.0),     # capture radius outside 3M
])
def test_schwarzschild(geon, compare, config, step, cap, pad, escape):
    m = geon.Schwarzschild(1.0, pad, escape)
    rng = np.random.default_rng(config)
    # everywhere, around 3M and the capture radius, and about to escape
    r = np.concatenate([rng.uniform(2.1, 50.0, 700), rng.uniform(2.005, 3.2, 300), escape * rng.uniform(0.99, 1.001, 100)])
    y = null_states("schwarzschild", r, rng, rng.uniform(size=len(r)) < 0.7)
    # next to the critical impact parameter, from 20M
    c = null_states("schwarzschild", np.full(200, 20.0), rng, True)
    s = 3.0 * np.sqrt(3.0) * np.sqrt(1.0 - 0.1) / 20.0
    a = np.arcsin(s * (1.0 + rng.normal(size=200) * 10.0 ** rng.uniform(-9, -1, 200)))
    c[:, 5], t = -np.cos(a) * np.sqrt(0.9), np.sin(a) / 20.0
    scale = t / np.hypot(c[:, 6], c[:, 7] * np.sin(c[:, 2]))
    c[:, 6] *= scale
    c[:, 7] *= scale
    timelike = null_states("schwarzschild", rng.uniform(4.0, 30.0, 64), rng, True)
    timelike[:, 4] *= 1.2
    radial = null_states("schwarzschild", rng.uniform(4.0, 30.0, 64), rng, True)
    radial[:, 6:] = 0.0
    y = np.concatenate([y, c, timelike, radial])
    if config in (SWEEP, SERVE_EQUATORIAL):
        y = on_equator(y)
    check(compare(m, config, y, step, cap), 0.3)


@pytest.mark.parametrize("config", [ORBIT, RENDER, SERVE_CAMERA])
@pytest.mark.parametrize("step,cap", [(0.05, 5000), (0.01, 1003), (0.7, 900), (-0.05, 905)])
def test_morris_thorne(geon, compare, config, step, cap):
    rng = np.random.default_rng(10 + config)
    # everywhere, the throat, and across |l| = 999 .. 1000
    r = np.concatenate([rng.uniform(-30.0, 30.0, 700), rng.uniform(-0.2, 0.2, 200), rng.uniform(998.5, 1000.2, 200),
                        -rng.uniform(998.5, 1000.2, 100)])
    y = null_states("morris_thorne", r, rng, rng.uniform(size=len(r)) < 0.5)
    y[:64, 6:] = 0.0
    y[64:128, 4] *= 1.3  # timelike
    check(compare(geon.MorrisThorne(1.0), config, y, step, cap))


@pytest.mark.parametrize("metric,config", [("schwarzschild", ORBIT), ("schwarzschild", SWEEP), ("schwarzschild", SERVE_EQUATORIAL),
                                           ("morris_thorne", ORBIT), ("morris_thorne", RENDER)])
def test_extreme_momenta(geon, compare, metric, config):
    """Momenta from 2^-140 to 2^120: doubled terms that leave the FP32 range first, and
    terms below it, with steps that move as far as ordinary ones do."""
    m = geon.Schwarzschild(1.0, 1.001, 60.0) if metric == "schwarzschild" else geon.MorrisThorne(1.0)
    rng = np.random.default_rng(77)
    y = null_states(metric, rng.uniform(2.01, 6.0, 4096), rng, rng.uniform(size=4096) < 0.5)
    if config in (SWEEP, SERVE_EQUATORIAL):
        y = on_equator(y)
    e = rng.integers(-140, 121, len(y))
    one = np.arange(len(y)) % 3
    y[one == 0, 4:] *= 2.0 ** e[one == 0, None]     # all of them
    y[one == 1, 7] *= 2.0 ** -np.abs(e[one == 1])   # nearly radial
    y[one == 1, 6] *= 2.0 ** -np.abs(e[one == 1])
    y[one == 2, 5] *= 2.0 ** -np.abs(e[one == 2])   # nearly tangential
    for step in (0.05, 2.0 ** -30, 2.0 ** -60, 2.0 ** 30):
        out = compare(m, config, y, step, 200)
        assert np.all(out[:, 0] == 0), (step, np.sum(out[:, 0] != 0), y[out[:, 0] != 0][:4])


def test_alcubierre_flat_groups(geon, compare):
    m = geon.Alcubierre(2.0, 0.25, 0.5, 0.0)
    rng = np.random.default_rng(4)
    n = 600
    y = np.zeros((n, 8))
    y[:, 1:4] = rng.uniform(-30.0, 30.0, (n, 3))
    y[:50, 1:4] = rng.uniform(-3.0, 3.0, (50, 3))
    d = rng.normal(size=(n, 3))
    y[:, 4], y[:, 5:] = 1.0, d / np.linalg.norm(d, axis=1)[:, None]
    y[100:200, 1:4] *= 33.0  # near the escape radius
    check(compare(m, CHART, y, 0.05, 4003))
