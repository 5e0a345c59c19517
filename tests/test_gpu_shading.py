"""What a ray's end is turned into: the sky on directions at the seams, of
extreme length and non-finite, against the oracle; the null residual against
the dense sum over all 16 entries of g in its order, also where p is not finite
(a zero entry times infinity is NaN there)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_sky_special_directions(geon, orc):
    vals = [0.0, -0.0, 1.0, -1.0, 0.6, -0.8, 1e-200, -1e-200, 1e200, -1e200, np.inf, -np.inf, np.nan]
    d = np.array([[a, b, c] for a in vals for b in vals for c in vals])
    for show in (True, False):
        assert np.array_equal(geon.sky.sample(d, show), orc.sky_sample(d, show))


@pytest.mark.parametrize("metric", ["minkowski", "schwarzschild", "alcubierre", "morris_thorne"])
def test_null_residual(geon, metric):
    m = {"minkowski": geon.Minkowski, "schwarzschild": geon.Schwarzschild, "alcubierre": geon.Alcubierre,
         "morris_thorne": geon.MorrisThorne}[metric]()
    rng = np.random.default_rng(6)
    n = 3000
    y = np.empty((n, 8))
    y[:, :4] = rng.uniform(0.2, 3.0, (n, 4))
    y[:, 4:] = rng.normal(size=(n, 4)) * 10.0 ** rng.uniform(-8, 8, (n, 1))
    y[:64, 4:] = 0.0
    for k, v in enumerate((np.inf, -np.inf, np.nan)):
        for a in range(4):
            y[100 + 4 * k + a, 4 + a] = v
    y[200:264, 4 + 2] = -0.0
    got = geon.trace(m, y, 0.05, 0).null_residual
    g = np.asarray(m.g(y[:, :4])).reshape(n, 16)
    s = np.zeros(n)
    with np.errstate(all="ignore"):
        for i in range(4):
            for j in range(4):
                s = s + g[:, 4 * i + j] * y[:, 4 + i] * y[:, 4 + j]
    assert np.array_equal(got, np.abs(s), equal_nan=True)
