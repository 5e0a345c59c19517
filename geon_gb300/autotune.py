"""Launch-configuration autotuner for the mixed-precision trace kernel.

The library times each register-cap variant of the kernel on a calibration
render of a metric and keeps the fastest for that metric kind
(geon_autotune_mixed). This module runs it, and remembers the result per GPU
model and build of the library in geon_gb300/_lib/autotune.json so later
processes skip the calibration.
"""
import ctypes
import hashlib
import json
import os

from . import _ffi
from ._util import check

CACHE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "_lib", "autotune.json")
CAPS = ("no register cap", "<=64 registers", "<=51 registers")
BLOCKS = (128, 64, 256)
# source 0 (camera rays, ray arrays): the register caps at 128 threads per block;
# source 1 (equatorial shadow rays): cap + 3 * block-size index, or BY_SIZE, the
# default: the kernel that suits the number of rays. The calibration leaves BY_SIZE
# unless a variant beats it, and sets that one for the sizes it was measured for.
VARIANTS = tuple(f"{c}, {b} threads/block" for b in BLOCKS for c in CAPS)
BY_SIZE = len(VARIANTS)


def _gpu_name():
    try:
        import torch
        return torch.cuda.get_device_name()
    except Exception:  # noqa: BLE001 - any failure just disables the cache key
        return "unknown-gpu"


def _build_id():
    """The built library: rates of another build say nothing about its kernels."""
    try:
        with open(_ffi.LIB_PATH, "rb") as f:
            return hashlib.sha256(f.read()).hexdigest()[:16]
    except OSError:
        return "unknown-build"


def block_size(variant):
    """Threads per block of an equatorial variant (None: by the number of rays, or not tuned)."""
    return BLOCKS[variant // len(CAPS)] if 0 <= variant < BY_SIZE else None


def _load():
    try:
        with open(CACHE) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}


def autotune(metric, n_rays=0, max_steps=20000, use_cache=True):
    """Pick the fastest variant per ray source for metric's kind.

    Returns {"variant": [camera/array source, equatorial source], "above": rays
    above which the equatorial variant holds, "rates": ...}.
    """
    lib = _ffi.load()
    key = (f"{_gpu_name()}|build={_build_id()}|kind={metric.kind}|rays={n_rays}|steps={max_steps}"
           f"|variants={len(VARIANTS)}")
    cache = _load() if use_cache else {}
    if key in cache:
        camera, equatorial = (int(v) for v in cache[key]["variant"])
        check(lib.geon_set_mixed_variant(metric.kind, 0, camera))
        if equatorial >= 0:
            check(lib.geon_set_sweep_variant_above(metric.kind, equatorial, int(cache[key]["above"])))
        return cache[key]
    rates = (ctypes.c_double * 12)()
    best = (ctypes.c_int * 2)()
    check(lib.geon_autotune_mixed(metric.handle, int(n_rays), int(max_steps), rates, best))
    entry = {"variant": [int(best[0]), int(best[1])], "above": int(lib.geon_get_sweep_variant_above(metric.kind)),
             "rates": {"camera": [float(r) for r in rates[:3]], "equatorial": [float(r) for r in rates[3:]]},
             "block_size": {"camera": 128, "equatorial": block_size(int(best[1]))},
             "variants": list(VARIANTS), "calibration": {"rays": int(n_rays), "max_steps": int(max_steps)}}
    if use_cache:
        cache[key] = entry
        try:
            os.makedirs(os.path.dirname(CACHE), exist_ok=True)
            with open(CACHE, "w") as f:
                json.dump(cache, f, indent=1)
        except OSError:
            pass
    return entry


def current_variant(kind, source=0):
    return _ffi.load().geon_get_mixed_variant(int(kind), int(source))
