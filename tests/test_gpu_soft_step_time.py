"""Rays for which the FP64 steps cannot run in the integer pipes (a momentum
component that is zero and stays so) take the FP64 pipe's step alone, not both."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rays(n, zero):
    rng = np.random.default_rng(1)
    y = np.zeros((n, 8))
    psi, alpha, r = rng.uniform(-1.0, 1.0, n), rng.uniform(0.2, 1.2, n), 30.0
    f = 1.0 - 2.0 / r
    y[:, 1], y[:, 2] = r, rng.uniform(1.0, 2.0, n)
    y[:, 4], y[:, 5] = 1.0 / np.sqrt(f), np.cos(alpha) * np.sqrt(f)
    y[:, 6] = np.sin(alpha) * np.sin(psi) / r
    y[:, 7] = np.sin(alpha) * np.cos(psi) / r / np.sin(y[:, 2])
    if zero == "meridional":
        y[:, 7] = 0.0
    elif zero == "radial":
        y[:, 6:] = 0.0
    elif zero == "one in 32":
        y[::32, 7] = 0.0
    return y


# The FP64 pipe's step takes 1.4 (FP64) and 1.5 (FP64_FAST) times as long as the
# integer step at these sizes, both steps 2.4; the bound lies between them.
@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
@pytest.mark.parametrize("zero", ["meridional", "radial", "one in 32"])
def test_one_step_not_both(geon, precision, zero):
    m = geon.Schwarzschild(1.0, 1.001, 1000.0)

    def best(y):
        times = []
        for _ in range(6):
            t = time.perf_counter()
            r = geon.trace(m, y, 0.05, 1200, precision=precision)
            times.append(time.perf_counter() - t)
        assert (r.steps_taken == 1200).all()
        return min(times)

    n = 36001
    assert best(rays(n, zero)) < 1.95 * best(rays(n, None))
