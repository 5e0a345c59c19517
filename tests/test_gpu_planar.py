"""The planar step with one combined test (mixed path, equatorial rays) against
the step with the separate tests, which the FP64-band option still runs (a band
no ray enters): the same classes, steps and final states, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r_obs,step,cap,metric", [
    (20.0, 0.01, 20000, (1.0, 1.001, 100.0)),   # the sweep's step
    (20.0, 0.05, 517, (1.0, 1.001, 1000.0)),    # ends at a cap off the group size
    (3.02, 0.02, 4000, (1.0, 1.001, 60.0)),     # starts at the photon sphere
    (2.3, 0.03, 3000, (1.0, 1.001, 40.0)),      # starts inside it
    (12.0, 0.5, 400, (1.0, 1.001, 50.0)),       # a step of half M: horizon and unresolved-infall rules
    (30.0, 0.05, 3000, (1.0, 1.8, 45.0)),       # capture radius outside 3M
    (50.0, 0.1, 2000, (2.5, 1.001, 30.0)),      # another mass
    (49.99, 0.05, 64, (1.0, 1.001, 50.0)),      # ends at the escape radius at once
    (20.0, -0.05, 900, (1.0, 1.001, 100.0)),    # backwards
])
def test_equals_separate_tests(geon, r_obs, step, cap, metric):
    m = geon.Schwarzschild(*metric)
    rng = np.random.default_rng(3)
    s = 3.0 * np.sqrt(3.0) * metric[0] * np.sqrt(max(0.0, 1.0 - 2.0 * metric[0] / r_obs)) / r_obs
    crit = np.arcsin(min(1.0, s))
    alpha = np.concatenate([rng.uniform(0.0, np.pi, 300), crit + rng.normal(size=100) * 10.0 ** rng.uniform(-12, -1, 100),
                            [0.0, np.pi / 2, np.pi]])
    lib = geon._load()
    fast = geon.shadow.trace(m, r_obs, alpha, step, cap, precision="mixed")
    term, steps = geon.shadow.classify(m, r_obs, alpha, step, cap, precision="mixed")
    lib.geon_set_mixed_band(1, 1e-6)
    try:
        plain = geon.shadow.trace(m, r_obs, alpha, step, cap, precision="mixed")
    finally:
        lib.geon_set_mixed_band(1, 0.0)
    assert np.array_equal(fast.termination, plain.termination) and np.array_equal(term, plain.termination)
    assert np.array_equal(fast.steps_taken, plain.steps_taken) and np.array_equal(steps, plain.steps_taken)
    assert np.array_equal(fast.final_state, plain.final_state, equal_nan=True)
