"""Launch variants of the mixed shadow sweep: one that is set runs at every number
of rays, the default goes by the number of rays, and the autotuner's choice holds
where it was measured. Host rule (sweep_rule.h), its C ABI, and on the GPU the same
results from every variant."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "geon_gb300", "csrc")
SMS = 152
ONE_WARP, HELD = SMS * 128, SMS * 1024
BY_SIZE, CHAIN, RESIDENT = 9, 10, 11


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    out = tmp_path_factory.mktemp("sweep_rule") / "librule.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-I{CSRC}",
                    os.path.join(ROOT, "tests", "sweep_rule_harness.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    ll, i = ctypes.c_longlong, ctypes.c_int
    lib.choice.restype, lib.choice.argtypes = ll, [i, ll]
    lib.chosen.argtypes = [ll, ll]
    lib.kernel.argtypes = [i, ll, i, i]
    lib.ordered.argtypes = [ll, i]
    lib.tuned.restype, lib.tuned.argtypes = ll, [ctypes.POINTER(ctypes.c_double), ll, i]
    return lib


@pytest.mark.parametrize("n", [1, ONE_WARP, ONE_WARP + 1, HELD, HELD + 1, 18 * ONE_WARP, 18 * ONE_WARP + 1, 1 << 33])
def test_set_variant_runs_at_every_size(rule, n):
    for v in range(9):
        assert rule.kernel(rule.chosen(rule.choice(v, 0), n), n, SMS, 0) == v
    fits = ONE_WARP < n <= HELD
    by_size = CHAIN if n <= ONE_WARP else RESIDENT if fits else 2 if n > 18 * ONE_WARP else 3
    assert rule.kernel(rule.chosen(rule.choice(BY_SIZE, 0), n), n, SMS, int(fits)) == by_size
    # a choice for more than HELD rays leaves the others to the rule
    assert rule.chosen(rule.choice(6, HELD), n) == (6 if n > HELD else BY_SIZE)


@pytest.mark.parametrize("n", [1000, HELD, HELD + 1, 466944])
def test_tuned_choice(rule, n):
    def tuned(rates):
        c = rule.tuned((ctypes.c_double * 9)(*rates), n, SMS)
        return rule.chosen(c, n), rule.chosen(c, HELD), rule.chosen(c, 1 << 40)
    queue = 2 if n > 18 * ONE_WARP else 3
    flat = [100.0] * 9
    assert tuned(flat) == (BY_SIZE,) * 3
    noise = list(flat)
    noise[6] = 101.9  # within 2 % of the kernel the rule runs
    assert tuned(noise) == (BY_SIZE,) * 3
    better = list(flat)
    better[6], better[7] = 110.0, 108.0
    # nothing is chosen at a size where the rule runs a kernel that was not timed
    assert tuned(better) == ((BY_SIZE,) * 3 if n <= HELD else (6, BY_SIZE, 6))
    better[queue] = 120.0
    assert tuned(better) == (BY_SIZE,) * 3


@pytest.mark.parametrize("n,ordered", [(1, 0), (2 * ONE_WARP, 0), (2 * ONE_WARP + 1, 1), (39500, 1), (1 << 20, 1),
                                       ((1 << 31) - 1, 1), (1 << 31, 0)])
def test_claim_order_from_the_third_warp(rule, n, ordered):
    assert rule.ordered(n, SMS) == ordered


def test_setters_without_gpu():
    import geon_gb300
    lib = geon_gb300._load()
    assert [lib.geon_get_mixed_variant(1, s) for s in (0, 1)] == [0, BY_SIZE]
    try:
        assert lib.geon_set_mixed_variant(1, 1, 4) == 0 and lib.geon_get_sweep_variant_above(1) == 0
        assert lib.geon_set_sweep_variant_above(1, 7, 1000) == 0
        assert lib.geon_get_mixed_variant(1, 1) == 7 and lib.geon_get_sweep_variant_above(1) == 1000
        for kind, v, above in [(1, 10, 0), (1, -1, 0), (1, 2, -1), (4, 2, 0)]:
            assert lib.geon_set_sweep_variant_above(kind, v, above) != 0
        assert lib.geon_set_mixed_variant(1, 1, 10) != 0 and lib.geon_set_mixed_variant(1, 0, 3) != 0
        assert lib.geon_get_mixed_variant(1, 1) == 7
    finally:
        lib.geon_set_mixed_variant(1, 1, BY_SIZE)


def test_cached_choice(monkeypatch, tmp_path):
    """A cached choice is applied with its range, and belongs to one build of the library."""
    import geon_gb300
    from geon_gb300 import autotune
    lib = geon_gb300._load()
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "autotune.json"))
    monkeypatch.setattr(autotune, "_gpu_name", lambda: "gpu")
    calls = []

    class Fake:  # the calibration itself needs a GPU
        def __getattr__(self, name):
            return getattr(lib, name)

        def geon_autotune_mixed(self, handle, n, steps, rates, best):
            calls.append(n)
            best[0], best[1] = 1, 6
            lib.geon_set_mixed_variant(1, 0, 1)
            return lib.geon_set_sweep_variant_above(1, 6, HELD)

    class Metric:
        kind, handle = 1, None
    monkeypatch.setattr(autotune._ffi, "load", lambda: Fake())
    try:
        first = autotune.autotune(Metric)
        assert first["variant"] == [1, 6] and first["above"] == HELD and first["block_size"]["equatorial"] == 256
        lib.geon_set_mixed_variant(1, 0, 0), lib.geon_set_mixed_variant(1, 1, BY_SIZE)
        assert autotune.autotune(Metric) == first and calls == [0]
        assert lib.geon_get_mixed_variant(1, 0) == 1 and lib.geon_get_mixed_variant(1, 1) == 6
        assert lib.geon_get_sweep_variant_above(1) == HELD
        monkeypatch.setattr(autotune, "_build_id", lambda: "another build")
        autotune.autotune(Metric)
        assert calls == [0, 0]
    finally:
        lib.geon_set_mixed_variant(1, 0, 0), lib.geon_set_mixed_variant(1, 1, BY_SIZE)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [700, ONE_WARP, 2 * ONE_WARP + 1, 60001, HELD + 1, 18 * ONE_WARP + 1])
def test_every_variant_gives_the_same_results(geon, n):
    m = geon.Schwarzschild(1.0, 1.001, 30.0)
    alpha = np.radians(np.random.default_rng(n).uniform(10.0, 20.0, n))
    lib = geon._load()
    term, steps = geon.shadow.classify(m, 20.0, alpha, 0.05, 1500, precision="mixed")
    try:
        for v in range(9):
            assert lib.geon_set_mixed_variant(1, 1, v) == 0
            t, s = geon.shadow.classify(m, 20.0, alpha, 0.05, 1500, precision="mixed")
            assert np.array_equal(t, term) and np.array_equal(s, steps)
    finally:
        lib.geon_set_mixed_variant(1, 1, BY_SIZE)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4096, 0])
def test_autotune_leaves_small_sweeps_to_the_rule(geon, n):
    from geon_gb300 import autotune
    lib = geon._load()
    try:
        r = autotune.autotune(geon.Schwarzschild(1.0, 1.001, 100.0), n_rays=n, max_steps=300, use_cache=False)
        assert all(x > 0.0 for x in r["rates"]["equatorial"])
        v, above = lib.geon_get_mixed_variant(1, 1), lib.geon_get_sweep_variant_above(1)
        assert v == r["variant"][1] == BY_SIZE or (n == 0 and above >= HELD)
    finally:
        lib.geon_set_mixed_variant(1, 0, 0), lib.geon_set_mixed_variant(1, 1, BY_SIZE)


@pytest.mark.gpu
def test_tuned_sweep_is_no_slower(geon):
    """What the autotuner chooses is measured on the sweeps' own claim order: it is not
    slower than the default on a large sweep (3 % for 256-thread blocks, measured)."""
    import time

    from geon_gb300 import autotune
    lib = geon._load()
    m = geon.Schwarzschild(1.0, 1.001, 1000.0)
    alpha = np.radians(np.random.default_rng(1).uniform(10.0, 20.0, 1 << 20))

    def best():
        times = []
        for _ in range(3):
            t = time.perf_counter()
            geon.shadow.classify(m, 20.0, alpha, 0.01, 200000, precision="mixed")
            times.append(time.perf_counter() - t)
        return min(times)

    try:
        default = best()
        autotune.autotune(m, use_cache=False)
        assert best() < 1.015 * default
    finally:
        lib.geon_set_mixed_variant(1, 0, 0), lib.geon_set_mixed_variant(1, 1, BY_SIZE)
