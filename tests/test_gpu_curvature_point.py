"""The curvature kernel with one thread per point (large batches) against the
oracle and against the cooperative kernel (small batches), bit for bit: every
output, ordinary points, and points where the metric or its symbols are not
finite (the horizon, the axis, a superluminal wall, far away)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 9473  # over the point kernel's threshold, not a multiple of its block
METRICS = [(2, (2.0, 0.5, 2.0, 0.0)), (2, (2.0, 0.125, 0.5, -0.3)), (3, (1.0,)), (3, (0.25,)), (1, (1.0, 1.001, 1000.0)),
           (1, (2.5, 1.001, 1000.0))]


def points(kind, params, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((N, 4))
    x[:, 0] = rng.uniform(-1.0, 1.0, N)
    if kind == 2:
        x[:, 1:] = rng.uniform(-4.0, 4.0, (N, 3))
        x[0, 1:] = 0.0                       # the bubble's centre
        x[1, 1:] = [params[3], 0.0, 0.0]
        x[2, 1:] = 1e3                       # flat
        x[3, 1:] = 1e160                     # r_s overflows
        x[4, 2] = np.nan
        x[5, 1] = np.inf
    else:
        x[:, 1] = rng.uniform(-5.0, 5.0, N) if kind == 3 else rng.uniform(0.5, 60.0, N)
        x[:, 2] = rng.uniform(-0.2, 3.4, N)
        x[:, 3] = rng.uniform(-7.0, 7.0, N)
        x[0, 2] = 0.0                        # the axis
        x[1, 2] = np.pi
        x[2, 1] = 2.0 * params[0]            # the horizon
        x[3, 1] = 0.0
        x[4, 1] = 1e160
        x[5, 2] = np.nan
        x[6, 1] = np.inf
        x[7, 2] = 1e9
        x[8, 2] = np.pi / 4
        x[9, 2] = 5.0 * np.pi / 4
    return x


@pytest.mark.parametrize("kind,params", METRICS)
@pytest.mark.parametrize("what", ["ricci", "ricci_scalar", "einstein", "stress_energy"])
def test_equals_cooperative_kernel(geon, kind, params, what):
    m = geon.from_kind(kind, params)
    x = points(kind, params, 5)
    f = getattr(geon.curvature, what)
    singular = []
    for i in range(16):
        try:
            f(m, x[i])
        except geon.GeonError as e:
            singular.append((i, e.status))
    if singular:  # the batch is refused as the point is
        with pytest.raises(geon.GeonError) as err:
            f(m, x)
        assert err.value.status == singular[0][1]
        x = np.concatenate([np.delete(x, [i for i, _ in singular], axis=0), x[-len(singular):]])
    parts = [f(m, x[q:q + 1000]) for q in range(0, N, 1000)]
    assert np.array_equal(f(m, x), np.concatenate(parts), equal_nan=True)


@pytest.mark.parametrize("kind,params", METRICS)
def test_equals_oracle(geon, orc, kind, params):
    m = geon.from_kind(kind, params)
    x = points(kind, params, 6)
    x[:16] = x[16:32]
    ref = orc.curvature(kind, list(params), x, "einstein", math=orc.GEON)
    assert np.array_equal(geon.curvature.einstein(m, x).reshape(N, -1), np.asarray(ref).reshape(N, -1), equal_nan=True)


@pytest.mark.parametrize("kind,params", METRICS)
@pytest.mark.parametrize("nk", [1, 16])
def test_contractions(geon, kind, params, nk):
    """T(k, k) for shared and for per-point vectors, and the grid job's vectors."""
    m = geon.from_kind(kind, params)
    x = points(kind, params, 7)
    x[:16] = x[16:32]
    rng = np.random.default_rng(8)
    for k in (rng.normal(size=(nk, 4)), rng.normal(size=(N, nk, 4))):
        whole = geon.curvature.nec_contraction(m, x, k)
        parts = [geon.curvature.nec_contraction(m, x[q:q + 1000], k if k.ndim == 2 else k[q:q + 1000])
                 for q in range(0, N, 1000)]
        assert np.array_equal(whole, np.concatenate(parts), equal_nan=True)
    lo, hi = ((-4.0, -4.0, -4.0), (4.0, 4.0, 4.0)) if kind == 2 else (
        (-3.0 if kind == 3 else 1.0, 0.1, 0.0), (9.0, 3.3, 6.0))
    n = (23, 21, 20)
    pts, ein, nec, kk = geon.curvature.grid(m, lo, hi, n, t=0.5, nk=nk, seed=99, with_k=True)
    e = [geon.curvature.einstein(m, pts[q:q + 1000]) for q in range(0, len(pts), 1000)]
    assert np.array_equal(ein, np.concatenate(e), equal_nan=True)
    t = [geon.curvature.nec_contraction(m, pts[q:q + 1000], kk[q:q + 1000]) for q in range(0, len(pts), 1000)]
    assert np.array_equal(nec, np.concatenate(t), equal_nan=True)
