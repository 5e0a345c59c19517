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


BOXES = [(1, (1.0, 1.001, 1000.0), (1e150, 0.1, 0.0), (1e160, 3.0, 6.0)),  # r^2 overflows: no tetrad
         (1, (1.0, 1.001, 1000.0), (1e-160, 0.1, 0.0), (1e-150, 3.0, 6.0)),
         (1, (1.0, 1.001, 1000.0), (0.5, 0.0, 0.0), (9.0, 3.141592653589793, 6.0)),  # the axis, inside the horizon
         (1, (1.0, 1.001, 1000.0), (1e70, 0.1, 0.0), (1e80, 3.0, 6.0)),
         (3, (1.0,), (-1e160, 0.1, 0.0), (1e160, 3.0, 6.0)), (3, (1.0,), (-1e90, 0.1, 0.0), (1e90, 3.0, 6.0)),
         (2, (2.0, 0.5, 5.0, 0.0), (-4.0,) * 3, (4.0,) * 3), (2, (2.0, 0.5, 1e60, 0.0), (-4.0,) * 3, (4.0,) * 3),
         (2, (2.0, 0.5, 0.8, 0.0), (-1e160,) * 3, (1e160,) * 3)]


@pytest.mark.parametrize("kind,params,lo,hi", BOXES)
def test_grid_vectors(geon, kind, params, lo, hi):
    """A grid against its slices along z as grids of their own (the cooperative
    kernel): Einstein tensors, which vectors are NaN, and the first slice's
    vectors and contractions."""
    m = geon.from_kind(kind, params)
    n, nk, seed = (24, 23, 22), 4, 99
    c = geon.curvature

    def f(lo, hi, n, seed):
        size = n[0] * n[1] * n[2]
        e, v, k = np.full((size, 16), 7.0), np.full((size, nk), 7.0), np.full((size, nk, 4), 7.0)
        rc = geon._load().geon_curvature_grid(m.handle, c._grid_desc(lo, hi, n, 0.5), nk, seed, dp(e), dp(v), dp(k))
        return rc, e, v, k

    rc, ein, nec, k = f(lo, hi, n, seed)
    z = c.grid_points(lo, hi, n)[::n[0] * n[1], 3]
    slice_points = n[0] * n[1]
    statuses = []
    for q in range(n[2]):
        # the vectors come from splitmix64(seed ^ (point * nk + q)): the first
        # slice's are the whole grid's
        at = slice(q * slice_points, (q + 1) * slice_points)
        s, e1, v1, k1 = f((lo[0], lo[1], z[q]), (hi[0], hi[1], z[q]), (n[0], n[1], 1), seed)
        statuses.append(s)
        assert np.array_equal(ein[at], e1, equal_nan=True)
        assert np.array_equal(np.isnan(k[at]).any(axis=2)[:, 0], np.isnan(k1).any(axis=2)[:, 0])
        if q == 0:
            assert np.array_equal(k[at], k1, equal_nan=True)
            assert np.array_equal(nec[at], v1, equal_nan=True)
    assert rc == min(statuses)
