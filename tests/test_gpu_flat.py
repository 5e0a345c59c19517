"""Groups of steps through the flat space around an Alcubierre bubble: the same
bits as the step-by-step trace. FP64 against the oracle; mixed against the step
restated in numpy for rays that move away from the bubble."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (radius, thickness, velocity, ship_x), step, steps: the reference's defaults, a
# thin wall, a wall at the limit of the rule and beyond it, a moved ship, a
# negative velocity, a backward step, a step longer than the bubble
CASES = [((2.0, 0.5, 2.0, 0.0), 0.05, 400), ((2.0, 0.125, 0.5, 0.0), 0.05, 999), ((2.0, 1e-4, 0.5, 3.0), 0.05, 333),
         ((2.0, 5e-5, 0.5, 0.0), 0.05, 100), ((1.0, 0.25, -0.7, -6.0), 0.1, 257), ((2.0, 0.125, 0.5, 0.0), -0.05, 160),
         ((0.5, 0.1, 0.9, 0.0), 30.0, 48)]


def rays(seed, n=192):
    """Rays that start inside, at the edge of and far from the bubble, some
    leaving the escape radius, with zero and non-null momenta among them."""
    rng = np.random.default_rng(seed)
    y = np.zeros((n, 8))
    r = np.concatenate([rng.uniform(0.0, 8.0, n // 3), rng.uniform(8.0, 60.0, n // 3), rng.uniform(980.0, 1001.0, n // 3)])
    d = rng.normal(size=(n, 3))
    y[:, 1:4] = r[:, None] * d / np.linalg.norm(d, axis=1)[:, None]
    y[:, 0] = rng.uniform(-1.0, 1.0, n)
    y[:, 4:] = rng.normal(size=(n, 4))
    y[::7, 5] = 0.0
    y[::11, 6] = -0.0
    y[0, 4:] = 0.0
    y[1, 5] = np.inf
    y[2, 4] = np.nan
    y[3, 0] = 1e300
    return y


@pytest.mark.parametrize("params,step,steps", CASES)
def test_fp64_equals_oracle(geon, orc, params, step, steps):
    y0 = rays(11)
    r = geon.trace(geon.Alcubierre(*params), y0, step, steps)
    term, yf, st, _ = orc.trace(2, list(params), y0, step, steps, math=orc.GEON)
    assert np.array_equal(r.termination, term) and np.array_equal(r.steps_taken, st)
    assert np.array_equal(r.final_state, yf, equal_nan=True)


def two_sum(hi, lo, inc):
    t = inc + lo
    s = hi + t
    bb = s - hi
    return s, (hi - (s - bb)) + (t - bb)


@pytest.mark.parametrize("params,step,steps", [c for c in CASES if c[1] < 1.0])
def test_mixed_equals_restatement(geon, params, step, steps):
    """Rays moving away from the bubble through flat space, off the group size,
    against the compensated FP32 step restated with zero derivatives."""
    rng = np.random.default_rng(5)
    n = 256
    d = rng.normal(size=(n, 3))
    d[::5, 2] = 0.0
    d /= np.linalg.norm(d, axis=1)[:, None]
    y0 = np.zeros((n, 8))
    r = params[0] + 9.6 * params[1] + 0.01 + rng.uniform(0.0, 400.0, n) * rng.uniform(0.0, 1.0, n) ** 4
    y0[:, 1:4] = r[:, None] * d
    y0[:, 1] += params[3]
    y0[:, 4] = 1.0
    y0[:, 5:] = np.sign(step) * d * rng.uniform(0.01, 1.5, n)[:, None]  # outward
    hi = y0.astype(np.float32)
    lo = (y0 - hi).astype(np.float32)
    h6 = np.float32(step / 6.0)
    two, zero = np.float32(2.0), np.float32(0.0)
    for _ in range(steps):
        p = hi[:, 4:]
        inc = h6 * ((two * p + (two * p + p)) + p)
        hi[:, :4], lo[:, :4], (hi[:, 4:], lo[:, 4:]) = (*two_sum(hi[:, :4], lo[:, :4], inc), two_sum(p, lo[:, 4:], zero))
    got = geon.trace(geon.Alcubierre(*params), y0, step, steps, precision="mixed")
    assert np.all(got.steps_taken == steps)
    assert np.array_equal(got.final_state, hi.astype(np.float64) + lo.astype(np.float64))
