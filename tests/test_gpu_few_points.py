"""dg and Christoffel symbols at few points (8 lanes per point) against the same
points inside a call above the size of that route (one thread per point): the
same bits, for whole and partial warps, every metric and non-finite inputs."""
import numpy as np
import pytest

from geon_gb300._util import dp

pytestmark = pytest.mark.gpu

FEW = 152 * 64


def metrics(geon):
    alc = geon.Alcubierre(2.0, 0.5, 2.0, 0.3)
    return {"schwarzschild": geon.Schwarzschild(1.0, 1.001, 100.0), "alcubierre": alc,
            "morris_thorne": geon.MorrisThorne(1.5),
            "field": geon.FieldMetric.sample(geon.Alcubierre(2.0, 0.5, 2.0, 0.0), [-4.0] * 3, [4.0] * 3, [17, 18, 19])}


@pytest.mark.parametrize("call", ["dg", "christoffel"])
@pytest.mark.parametrize("metric", ["schwarzschild", "alcubierre", "morris_thorne", "field"])
def test_same_bits(geon, metric, call):
    m = metrics(geon)[metric]
    rng = np.random.default_rng(11)
    x = rng.uniform(-5.0, 5.0, (FEW + 1, 4))
    if metric in ("schwarzschild", "morris_thorne"):
        x[:, 2] = rng.uniform(0.1, 3.0, FEW + 1)
    x[0] = [0.0, 0.3, 0.0, 0.0]  # the bubble's centre
    x[2, 1:] = 1e-9
    x[4, 1] = 1e150
    x[5, 0] = 1e12  # a t that a step of the differences does not change

    def f(points):  # status and values: the wormhole's axis (first point) is singular, and its values are written
        out = np.full((len(points), 64), 7.0)
        return getattr(geon._load(), "geon_metric_" + call)(m.handle, dp(points), len(points), dp(out)), out

    status, whole = f(x)
    assert status == (-2 if (metric, call) == ("morris_thorne", "christoffel") else 0)
    for n in (1, 2, 3, 4, 5, 7, 33, 1000, FEW):
        rc, out = f(x[:n])
        assert rc == status
        assert np.array_equal(out, whole[:n], equal_nan=True), n


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("metric", ["schwarzschild", "alcubierre", "morris_thorne", "field"])
def test_nonfinite(geon, metric, value):
    m = metrics(geon)[metric]
    x = np.tile([0.5, 3.0, 1.0, 2.0], (FEW + 1, 1))
    for a in range(4):
        x[a, a] = value
    for call in ("dg", "christoffel"):
        f = getattr(m, call)
        whole = status = None
        try:
            whole = np.asarray(f(x))
        except geon.GeonError as e:
            status = e.status
        if whole is None:
            with pytest.raises(geon.GeonError) as err:
                f(x[:5])
            assert err.value.status == status
        else:
            assert np.array_equal(np.asarray(f(x[:5])), whole[:5], equal_nan=True), call


def test_singular(geon):
    m = geon.MorrisThorne(1.0)
    x = np.tile([0.0, 1.0, 1.0, 0.0], (6, 1))
    m.christoffel(x)
    x[5, 2] = 0.0
    with pytest.raises(geon.GeonError) as e:
        m.christoffel(x)
    assert e.value.status == -2
