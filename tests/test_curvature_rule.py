"""The choice between the two curvature kernels: against measured times (the
slower kernel is never chosen by much), and, on the GPU, the same bits on both sides
of every line of the rule."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from geon_gb300._util import dp

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "geon_gb300", "csrc")
SMS = 152

# (Alcubierre, grid, points, vectors, us with one thread per point, us of the block kernel) on 152 SMs
MEASURED = [
    (1, 1, 9261, 0, 222.7, 177.7), (1, 1, 9261, 16, 288.8, 213.0), (1, 1, 13824, 0, 236.5, 190.5),
    (1, 1, 13824, 16, 309.2, 251.9), (1, 1, 19683, 0, 233.5, 281.6), (1, 1, 19683, 16, 306.2, 366.6),
    (1, 1, 28830, 16, 329.8, 525.3), (1, 1, 64000, 16, 699.9, 1258.0), (1, 1, 9728, 256, 1096.2, 794.1),
    (1, 1, 14592, 1024, 4541.4, 4096.0), (1, 1, 19456, 1024, 4551.7, 5455.4),
    (1, 0, 9728, 0, 269.8, 168.1), (1, 0, 9728, 16, 315.4, 202.6), (1, 0, 14592, 0, 278.3, 170.6),
    (1, 0, 14592, 256, 911.0, 686.6), (1, 0, 19456, 16, 335.7, 281.5), (1, 0, 24320, 16, 362.9, 351.2),
    (1, 0, 38912, 0, 371.2, 419.9), (1, 0, 116736, 16, 1187.3, 1357.0),
    (0, 1, 5120, 0, 34.1, 78.7), (0, 1, 5168, 16, 93.2, 108.5), (0, 1, 6080, 64, 270.3, 200.7),
    (0, 1, 6080, 256, 981.5, 568.8), (0, 1, 9728, 16, 93.2, 138.2), (0, 1, 9728, 256, 981.5, 753.2),
    (0, 1, 14592, 64, 306.2, 394.2), (0, 1, 14592, 1024, 4371.5, 4077.6), (0, 1, 19456, 1024, 4372.5, 5425.7),
    (0, 0, 6080, 16, 103.0, 111.0), (0, 0, 6080, 64, 197.0, 151.0), (0, 0, 10000, 0, 77.0, 122.0),
    (0, 0, 14000, 100, 329.8, 352.7), (0, 0, 12288, 64, 241.5, 253.2), (0, 0, 10000, 64, 233.0, 222.0),
    (0, 0, 10000, 256, 685.0, 511.0), (0, 0, 12288, 256, 710.0, 609.0), (0, 0, 19456, 256, 789.0, 824.0),
]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    out = tmp_path_factory.mktemp("curvature_rule") / "librule.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-I{CSRC}",
                    os.path.join(ROOT, "tests", "curvature_rule_harness.cpp"), "-o", str(out)], check=True)
    f = ctypes.CDLL(str(out)).point_kernel
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
    return f


@pytest.mark.parametrize("alc,grid,n,nk,point,block", MEASURED)
def test_follows_the_measurements(rule, alc, grid, n, nk, point, block):
    chosen = point if rule(alc, grid, n, nk, SMS) else block
    assert chosen <= 1.06 * min(point, block)


def points(kind, n, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((n, 4))
    if kind == 2:
        x[:, 1:] = rng.uniform(-4.0, 4.0, (n, 3))
        edges = [[0, 0, 0, 0], [0, 1e3, 1e3, 1e3], [0, 1e160, 0, 0], [0, 1, np.nan, 0], [0, np.inf, 0, 0]]
    else:
        x[:, 1] = rng.uniform(2.5, 60.0, n)
        x[:, 2] = rng.uniform(-0.2, 3.4, n)
        x[:, 3] = rng.uniform(-7.0, 7.0, n)
        edges = [[0, 5, 1e-3, 0], [0, 1e160, 1, 0], [0, 5, np.nan, 0], [0, np.inf, 1, 0], [0, 5, np.pi / 4, 0]]
    x[7:12] = edges
    return x


KINDS = [(1, (1.0, 1.001, 1000.0)), (2, (2.0, 0.125, 0.5, -0.3)), (3, (1.0,))]
WIDTH = {"ricci": 16, "ricci_scalar": 1, "einstein": 16, "stress_energy": 16, "nec_contraction": None}


@pytest.mark.gpu
@pytest.mark.parametrize("kind,params", KINDS)
@pytest.mark.parametrize("op", list(WIDTH))
def test_batches_on_both_sides(geon, kind, params, op):
    m = geon.from_kind(kind, params)
    rng = np.random.default_rng(8)

    def f(x, k, shared):
        w = WIDTH[op] or k.shape[-2]
        out = np.full((len(x), w), 7.0)
        vectors = (dp(k), k.shape[-2], shared) if WIDTH[op] is None else ()
        return getattr(geon._load(), "geon_" + op)(m.handle, dp(x), len(x), *vectors, dp(out)), out

    sizes = [(33 * SMS - 1, 3), (33 * SMS, 3), (33 * SMS, 200)] if kind != 2 else [(128 * SMS, 3), (128 * SMS + 1, 3)]
    for n, nk in sizes + [(128 * SMS + 77, 40)]:
        x = points(kind, n, n)
        for shared in ((1,) if WIDTH[op] else (1, 0)):
            k = rng.normal(size=(nk, 4) if shared else (n, nk, 4))
            status, whole = f(x, k, shared)
            cut = range(0, n, 1500)
            parts = [f(np.ascontiguousarray(x[q:q + 1500]), k if shared else np.ascontiguousarray(k[q:q + 1500]), shared)
                     for q in cut]
            assert status == min(rc for rc, _ in parts)
            assert np.array_equal(whole, np.concatenate([v for _, v in parts]), equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,params", KINDS)
@pytest.mark.parametrize("shape,nk", [((17, 19, 16), 3), ((17, 19, 16), 130), ((24, 32, 19), 5), ((24, 32, 19), 90),
                                      ((25, 24, 25), 5), ((25, 24, 25), 150)])
def test_grids_on_both_sides(geon, kind, params, shape, nk):
    """A grid against its slices along z: Einstein tensors, and the first slice's vectors."""
    m = geon.from_kind(kind, params)
    lo, hi = ((-4.0,) * 3, (4.0,) * 3) if kind == 2 else ((2.5, 0.3, 0.0), (9.0, 2.8, 6.0))
    c = geon.curvature
    x, ein, nec, k = c.grid(m, lo, hi, shape, nk=nk, seed=5, with_k=True)
    per = shape[0] * shape[1]
    for q, z in enumerate(x[::per, 3]):
        at = slice(q * per, (q + 1) * per)
        _, e1, v1, k1 = c.grid(m, (*lo[:2], z), (*hi[:2], z), (*shape[:2], 1), nk=nk, seed=5, with_k=True)
        assert np.array_equal(ein[at], e1)
        if q == 0:
            assert np.array_equal(k[at], k1) and np.array_equal(nec[at], v1)
