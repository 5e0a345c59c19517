"""Point calls that go over as one block and calls just above that size give the
same bits, with a flagged point and with per-point directions."""
import numpy as np
import pytest

from geon_gb300.curvature import nec_contraction

pytestmark = pytest.mark.gpu

SMALL = 16384  # bytes of results, flags and inputs


def edge(per_point, fixed=8):
    """Most points whose block still fits."""
    return (SMALL - fixed) // per_point


@pytest.mark.parametrize("call,width", [("christoffel", 64), ("g", 16), ("g_inv", 16), ("dg", 64)])
@pytest.mark.parametrize("metric", ["alcubierre", "schwarzschild"])
def test_both_sides_of_the_size(geon, metric, call, width):
    m = geon.Alcubierre(2.0, 0.5, 2.0, 0.0) if metric == "alcubierre" else geon.Schwarzschild(1.0, 1.001, 100.0)
    n = edge(8 * (4 + width))
    rng = np.random.default_rng(3)
    x = rng.uniform(1.0, 3.0, (n + 1, 4))
    whole = np.asarray(getattr(m, call)(x))  # one point too many
    for k in (1, 2, n - 1, n):
        part = np.asarray(getattr(m, call)(x[:k]))
        assert np.array_equal(part, whole[:k])


def test_terminate_odd_counts(geon):
    m = geon.Schwarzschild(1.0, 1.001, 100.0)
    n = 600  # results padded to whole words; above 455 points the call is a large one
    x = np.zeros((n, 4))
    x[:, 1] = np.linspace(1.5, 150.0, n)
    x[:, 2] = 1.0
    whole = np.asarray(m.terminate(x))
    assert len(set(whole.tolist())) > 1
    for k in (1, 3, 453, 454, 455, 456):
        assert np.array_equal(np.asarray(m.terminate(x[:k])), whole[:k])


def test_singular_point(geon):
    """theta = 0 on the wormhole: g_phiphi = 0 and the call reports it at either size."""
    m = geon.MorrisThorne(1.0)
    for n in (1, 400):
        x = np.tile([0.0, 1.0, 1.0, 0.0], (n, 1))
        m.christoffel(x)
        x[-1, 2] = 0.0
        with pytest.raises(geon.GeonError):
            m.christoffel(x)


def test_directions_per_point(geon):
    """Null-energy contraction: inputs in two pieces, shared and per point."""
    m = geon.Alcubierre(2.0, 0.5, 2.0, 0.0)
    rng = np.random.default_rng(4)
    n, nk = 100, 3  # per point 32 + 96 + 24 bytes: 100 points fit, 120 do not
    x = rng.uniform(1.0, 3.0, (120, 4))
    k = rng.uniform(-1.0, 1.0, (120, nk, 4))
    whole = np.asarray(nec_contraction(m, x, k))
    assert np.array_equal(np.asarray(nec_contraction(m, x[:n], k[:n])), whole[:n])
    assert np.array_equal(np.asarray(nec_contraction(m, x[:1], k[:1])), whole[:1])
    shared = np.asarray(nec_contraction(m, x[:5], k[0]))
    each = np.asarray(nec_contraction(m, x[:5], np.repeat(k[:1], 5, axis=0)))
    assert np.array_equal(shared, each)
