"""Shadow sweeps over the sizes where the launch changes (one warp per SM
quarter, claim order, everything resident, the queue): every ray's class and
steps are those of the same rays in pieces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152  # GB300; other devices only move the edges


@pytest.mark.parametrize("n", [1, 31, 33, SMS * 128, SMS * 128 + 1, 39999, 40000, SMS * 1024 - 33, SMS * 1024,
                               SMS * 1024 + 1, SMS * 1152 + 1, 200003])
def test_sweep_equals_pieces(geon, n):
    m = geon.Schwarzschild(1.0, 1.001, 30.0)
    alpha = np.radians(np.random.default_rng(n).uniform(10.0, 20.0, n))
    term, steps = geon.shadow.classify(m, 20.0, alpha, 0.05, 3000, precision="mixed")
    parts = [geon.shadow.classify(m, 20.0, alpha[q:q + 15000], 0.05, 3000, precision="mixed") for q in range(0, n, 15000)]
    assert np.array_equal(term, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(steps, np.concatenate([p[1] for p in parts]))
