"""Curvature where finite Christoffel symbols overflow in the sums of the Ricci
tensor: large batches (one thread per point) against the same points in batches
of the cooperative kernel, bit for bit, non-finite entries included."""
import numpy as np
import pytest

from geon_gb300._util import dp

pytestmark = pytest.mark.gpu

N = 9473  # over the point kernel's threshold


def points(what):
    x = np.zeros((N, 4))
    x[:, 2] = 1.0
    if what == "radius":
        x[:, 1] = np.logspace(-170, 170, N)
    elif what == "near zero":
        x[:, 1] = np.linspace(0.5e-100, 2e-100, N)  # symbols up to 1e301, products of them infinite
    else:
        x[:, 1] = np.random.default_rng(3).uniform(-4.0, 4.0, N)
        x[:, 3] = np.random.default_rng(4).uniform(-4.0, 4.0, N)
    return x


WIDTH = {"ricci": 16, "ricci_scalar": 1, "einstein": 16, "stress_energy": 16, "nec_contraction": 3}


@pytest.mark.parametrize("kind,params,what", [
    (1, (1.0, 1.001, 1000.0), "radius"), (1, (1.0, 1.001, 1000.0), "near zero"), (3, (1.0,), "radius"),
    (2, (2.0, 0.5, 2.0, 0.0), "radius"), (2, (2.0, 0.5, 1e60, 0.0), "box"), (2, (2.0, 0.5, 1e100, 0.0), "box")])
@pytest.mark.parametrize("op", list(WIDTH))
def test_equals_cooperative_kernel(geon, kind, params, what, op):
    m = geon.from_kind(kind, params)
    x = points(what)
    k = np.random.default_rng(5).normal(size=(3, 4))

    def f(p):  # status and values: they are written where the metric is singular too
        out = np.full((len(p), WIDTH[op]), 7.0)
        vectors = (dp(k), 3, 1) if op == "nec_contraction" else ()
        return getattr(geon._load(), "geon_" + op)(m.handle, dp(p), len(p), *vectors, dp(out)), out

    status, whole = f(x)
    parts = [f(x[q:q + 1000]) for q in range(0, N, 1000)]
    assert status == min(rc for rc, _ in parts)
    assert np.array_equal(whole, np.concatenate([v for _, v in parts]), equal_nan=True)
