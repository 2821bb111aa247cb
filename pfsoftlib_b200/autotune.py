"""Project autotuner for the batched engine.

For a multiset of bandwidths ``tune_plan`` times, per bandwidth, the DWT of a PFSOFT_BATCH_SPLIT plan on
the split-precision kernel and on the FP64 kernels with CUDA events, caches the winners in a JSON
table keyed by GPU name and the sorted bandwidth counts, applies them to the library
(pfsoft_tune_split_bandwidth) and returns them. What else earlier kernels left to choose
(``transforms_per_cta``, pfsoft_tune_fft_fused) has no effect in the present ones: ``tune_batch`` and
the ``fft_fused`` entries keep their form, and nothing is timed for them.

``choose`` is the pure decision rule (tested on CPU).
"""
from __future__ import annotations

import ctypes
import json
import os
from collections import Counter

CANDIDATES = (1, 2, 4)


def cache_path() -> str:
    d = os.environ.get("PFSOFT_B200_CACHE", os.path.join(os.path.expanduser("~"), ".cache", "pfsoft_b200"))
    return os.path.join(d, "autotune.json")


def key_for(gpu: str, bandwidths) -> str:
    c = Counter(int(b) for b in bandwidths)
    return gpu + "|" + ",".join(f"{b}x{c[b]}" for b in sorted(c))


def choose(timings: dict) -> int:
    """The fastest candidate; ties go to the smaller value (less register and idle-warp cost)."""
    if not timings:
        raise ValueError("no timings")
    return min(sorted(timings), key=lambda k: (timings[k], k))


def load_cache(path: str | None = None) -> dict:
    path = path or cache_path()
    try:
        with open(path) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}


def store(key: str, value: int, path: str | None = None) -> None:
    path = path or cache_path()
    data = load_cache(path)
    data[key] = value
    try:
        os.makedirs(os.path.dirname(path), exist_ok=True)
        with open(path + ".tmp", "w") as f:
            json.dump(data, f, indent=1, sort_keys=True)
        os.replace(path + ".tmp", path)
    except OSError:
        pass


def tune_batch(lib, bandwidths, coeffs, grids, back, reps: int = 2, use_cache: bool = True) -> tuple[int, dict]:
    """The transforms-per-CTA argument of a batch plan and the timings in ms behind the choice. The kernels
    take one transform per CTA whatever it is, so the smallest candidate is returned, without timings."""
    return CANDIDATES[0], {}


def _time_ms(fn, reps: int) -> float:
    import torch

    fn()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        fn()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / reps


def apply(lib, plan: dict) -> None:
    """Sets the library's per-bandwidth knobs from a plan returned by tune_plan."""
    for b, on in plan.get("fft_fused", {}).items():
        lib.pfsoft_tune_fft_fused(int(b), int(bool(on)))
    for b, on in plan.get("split", {}).items():
        lib.pfsoft_tune_split_bandwidth(int(b), int(bool(on)))


def tune_plan(lib, bandwidths, coeffs, grids, back, reps: int = 2, use_cache: bool = True) -> dict:
    """Per distinct bandwidth of the mix: the DWT of a split plan on the split kernel or the FP64 kernels,
    timed on a batch plan of that bandwidth's transforms. Applies the winners (apply) and returns
    {"fft_fused": {B: False}, "split": {B: bool}, "ms": {"fft": {}, "dwt": {...}}}.
    Buffers are lists of CUDA tensors in the order of `bandwidths`."""
    import torch

    gpu = torch.cuda.get_device_name()
    key = "plan|" + key_for(gpu, bandwidths)
    if use_cache:
        cached = load_cache().get(key)
        if isinstance(cached, dict) and "fft_fused" in cached and "split" in cached:
            apply(lib, cached)
            return cached
    s = torch.cuda.current_stream().cuda_stream
    out = {"fft_fused": {}, "split": {}, "ms": {"fft": {}, "dwt": {}}}
    for b in sorted(set(int(x) for x in bandwidths)):
        idx = [i for i, x in enumerate(bandwidths) if int(x) == b]
        out["fft_fused"][str(b)] = False
        arr = (ctypes.c_int * len(idx))(*[b] * len(idx))
        cp = (ctypes.c_void_p * len(idx))(*[coeffs[i].data_ptr() for i in idx])
        gp = (ctypes.c_void_p * len(idx))(*[grids[i].data_ptr() for i in idx])
        bp = (ctypes.c_void_p * len(idx))(*[back[i].data_ptr() for i in idx])
        d = {}
        for flags in (0, 2):
            lib.pfsoft_tune_split_bandwidth(b, 1)
            plan = ctypes.c_void_p()
            if lib.pfsoft_batch_create(arr, len(idx), 0, flags | 1, ctypes.byref(plan)) != 0:
                continue
            try:
                d[flags] = _time_ms(lambda: (lib.pfsoft_batch_idsoft(plan, cp, gp, s),
                                             lib.pfsoft_batch_dsoft(plan, gp, bp, s)), reps)
            finally:
                lib.pfsoft_batch_destroy(plan)
        split = 2 in d and (0 not in d or d[2] <= d[0])
        lib.pfsoft_tune_split_bandwidth(b, int(split))
        out["split"][str(b)] = split
        out["ms"]["dwt"][str(b)] = {"split": d.get(2), "fp64": d.get(0), "transforms": len(idx)}
    store(key, out)
    return out
