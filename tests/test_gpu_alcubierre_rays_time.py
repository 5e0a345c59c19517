"""FP64 rays around a warp bubble whose wall they do not leave: the warps of a full
GPU must not wait for one another's instructions (the step has to fit the
instruction cache)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def best(geon, m, n):
    rng = np.random.default_rng(0)
    y = np.zeros((n, 8))
    y[:, 1], y[:, 4] = -10.0 * rng.uniform(0.8, 1.0, n), 1.02
    d = rng.normal(size=(n, 3))
    y[:, 5:] = d / np.linalg.norm(d, axis=1)[:, None]
    times = []
    for _ in range(4):
        t = time.perf_counter()
        geon.trace(m, y, 0.05, 400)
        times.append(time.perf_counter() - t)
    return min(times)


def test_one_warp_per_quarter_takes_as_long_as_a_few(geon):
    # 19456 rays are one warp on each of 608 SM quarters. Their FP64 operations, 4 warps
    # per SM at 16 cycles an instruction, stay below the chain of one warp's (64 cycles),
    # so they take little longer than 2000 rays do (measured: 72 and 61 ms; 142 and 80
    # with a step that outgrows the instruction cache).
    m = geon.Alcubierre(2.0, 0.5, 0.5, 0.0)
    assert best(geon, m, 19456) < 1.45 * best(geon, m, 2000)
