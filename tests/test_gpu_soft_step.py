"""FP64 Schwarzschild steps whose multiplications run in the integer pipes: the
oracle's bits on rays at the edges of their range, and, for both FP64 modes, the
bits of the same step on the FP64 pipe. The latter runs when an operand is
outside the range: momenta times 2^180 with steps times 2^-180 trace the same
points with every operation scaled exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rays(seed, n, equatorial):
    rng = np.random.default_rng(seed)
    y = np.zeros((n, 8))
    y[:, 0] = rng.uniform(-1.0, 1.0, n)
    y[:, 1] = rng.uniform(2.2, 40.0, n)
    y[:, 2] = np.pi / 2 if equatorial else rng.uniform(0.02, 3.12, n)
    y[:, 3] = rng.uniform(-3.0, 3.0, n)
    y[:, 4] = rng.uniform(0.5, 2.0, n)
    y[:, 5] = rng.uniform(-1.5, 1.0, n)
    if not equatorial:
        y[:, 6] = rng.normal(size=n) * 0.05
    y[:, 7] = rng.normal(size=n) * 0.1
    return y


@pytest.mark.parametrize("step,cap", [(0.05, 300), (0.01, 65), (1.0, 60)])
def test_edges_equal_oracle(geon, orc, step, cap):
    y = rays(1, 256, False)
    y[0, 4:] = 0.0
    y[1:9, 5], y[9:17, 6], y[17:25, 7] = 0.0, 0.0, 0.0   # zero operands
    y[25:33, 2] = [0.0, 1e-9, 1e-300, np.pi, 3.9, 3.95, -0.3, 50.0]
    y[33:37, 2] = [np.pi / 4, 3 * np.pi / 4, np.pi / 2, np.nan]
    y[37:41, 1] = [2.0, 2.0 + 1e-12, 1.0, np.inf]
    y[41:49, 4:] *= 2.0 ** np.array([-175, -169, -100, 100, 160, 169, 175, 400])[:, None]
    y[49:53, 6] = [1e-60, 1e-52, 1e-200, 1e-310]
    params = [1.0, 1.001, 100.0]
    r = geon.trace(geon.Schwarzschild(*params), y, step, cap)
    term, yf, steps, _ = orc.trace(1, params, y, step, cap, math=orc.GEON)
    assert np.array_equal(r.termination, term) and np.array_equal(r.steps_taken, steps)
    assert np.array_equal(r.final_state, yf, equal_nan=True)


@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
@pytest.mark.parametrize("equatorial", [False, True])
@pytest.mark.parametrize("mass,step,cap", [(1.0, 0.05, 1500), (0.7, 0.3, 400)])
def test_integer_and_fp64_pipe_agree(geon, precision, equatorial, mass, step, cap):
    m = geon.Schwarzschild(mass, 1.001, 60.0)
    y = rays(2, 512, equatorial)
    a = geon.trace(m, y, step, cap, precision=precision)
    s = 2.0 ** 180
    z = y.copy()
    z[:, 4:] *= s
    b = geon.trace(m, z, step / s, cap, precision=precision)
    # a ray flung off at the horizon to 1e100 and beyond overflows when scaled
    k = ~(np.abs(a.final_state).max(axis=1) > 1e100)
    assert np.sum(~k) <= 4
    assert np.array_equal(a.termination[k], b.termination[k]) and np.array_equal(a.steps_taken[k], b.steps_taken[k])
    assert np.array_equal(a.final_state[k, :4], b.final_state[k, :4], equal_nan=True)
    assert np.array_equal(a.final_state[k, 4:] * s, b.final_state[k, 4:], equal_nan=True)
