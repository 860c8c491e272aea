"""Autotuners of the step kernel and of the electrogram contraction.

Times every compiled step-kernel variant (voxels per thread, i.e. the tile
length of 256 x VPT voxels, and register budget) at every feasible
CTAs-per-SM setting on the engine's live instances, keeps the fastest (the
first option within 1 % of the fastest median, so near-ties resolve the same
way every run) and leaves the engine configured with it.  Each option is timed ``repeats`` times
(one launch of ``steps`` steps each, after a warm launch that also captures
its graph) and ranked by the median.  Tuning advances the instances like any
other call (the steps are real work).

Results are cached per GPU name, library (a digest of its file: a choice holds
for the kernels it was measured with) and workload bucket (precision, total voxels
rounded to a power of two, instance count): in the process, and in a JSON file
(``PHS_AUTOTUNE_CACHE``, default ``~/.cache/pyheartsim_b200/autotune.json``)
so later processes on the same machine start from the same choice.

:func:`tune_electrogram` picks the tile configuration (output tile 128 x 128,
128 x 256 or 256 x 256 by CTA pairs, K stage width and depth) of the BF16x3 electrogram contraction.
"""
import json
import math
import os

import torch

from . import _lib
from .engine import step_variants

_CACHE = {}
TIE_FRAC = 0.01


def cache_path():
    return os.environ.get("PHS_AUTOTUNE_CACHE") or os.path.join(os.path.expanduser("~"), ".cache", "pyheartsim_b200",
                                                                "autotune.json")


def _load_file():
    try:
        with open(cache_path()) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}


def _store_file(key, best):
    path = cache_path()
    try:
        data = _load_file()
        data[key] = list(best)
        os.makedirs(os.path.dirname(path), exist_ok=True)
        tmp = path + f".{os.getpid()}.tmp"
        with open(tmp, "w") as f:
            json.dump(data, f, indent=1, sort_keys=True)
        os.replace(tmp, path)
    except OSError:
        pass                                   # a read-only home: the in-process cache still works


def _bucket(engine):
    n = sum(engine.instance(s).n_voxel for s in engine.slots())
    return "|".join(str(x) for x in (torch.cuda.get_device_name(), _lib.revision(), engine.precision,
                                      1 << max(0, int(math.log2(max(n, 1)))), len(engine.slots())))


def tune(engine, steps=10, stream=None, cps_options=None, repeats=5, use_file=True):
    """Pick (variant, ctas_per_sm) for ``engine``; returns the timing table."""
    key = _bucket(engine)
    if key not in _CACHE and use_file:
        hit = _load_file().get(key)
        if hit is not None:
            _CACHE[key] = tuple(hit)
    if key in _CACHE:
        best = _CACHE[key]
        engine.configure(variant=best[0], ctas_per_sm=best[1])
        return {"cached": True, "best": best}
    stream = stream or torch.cuda.current_stream()
    table = []
    for variant, minb, regs, vpt in step_variants(engine.precision, with_vpt=True):
        options = cps_options or sorted({minb, max(1, minb - 1), minb + 1})
        for cps in options:
            engine.configure(variant=variant, ctas_per_sm=cps)
            try:
                engine.advance(steps, stream=stream, sync=True)      # plan + graph capture, warm
            except _lib.PhsError:
                continue
            times = []
            for _ in range(max(1, repeats)):
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                engine.advance(steps, stream=stream, sync=False)
                e1.record(stream)
                torch.cuda.synchronize()
                times.append(e0.elapsed_time(e1) / steps)
            times.sort()
            table.append({"variant": variant, "voxels_per_thread": vpt, "min_ctas": minb, "regs": regs,
                          "ctas_per_sm": cps, "ms_per_step": times[len(times) // 2],
                          "ms_per_step_min": times[0], "ms_per_step_max": times[-1]})
    # the first option (variant, then CTAs per SM, ascending) within TIE_FRAC
    # of the fastest median: options that differ by less than the run-to-run
    # spread do not flip the choice between runs
    fastest = min(r["ms_per_step"] for r in table)
    best = next(r for r in table if r["ms_per_step"] <= fastest * (1.0 + TIE_FRAC))
    _CACHE[key] = (best["variant"], best["ctas_per_sm"])
    if use_file:
        _store_file(key, _CACHE[key])
    engine.configure(variant=best["variant"], ctas_per_sm=best["ctas_per_sm"])
    return {"cached": False, "best": (best["variant"], best["ctas_per_sm"]), "table": table}


_EGM_CACHE = {}
EGM_TILE_NAMES = ("128x128 BK64 x3", "128x256 BK64 x2", "128x256 BK32 x4", "256x256 BK64 x3 (CTA pairs)")


def tune_electrogram(T, n_e, T_pad, E_pad, K_pad, vh, vl, mh, ml, out, work, stream=None, repeats=3):
    """Pick the tcgen05 tile configuration of the BF16x3 electrogram contraction
    (``phs_egm_contract_bf16x3_cfg``) for this shape: every configuration is
    run once to warm up, then timed ``repeats`` times (CUDA events on the
    stream) and ranked by the median.  The operands are device tensors (the
    split V and M), ``out`` the (T, n_e) FP32 result and ``work`` the workspace.
    Cached per GPU name and padded shape.  Returns (best config, {config:
    median ms})."""
    import ctypes
    key = (torch.cuda.get_device_name(), int(T_pad), int(E_pad), int(K_pad))
    if key in _EGM_CACHE:
        return _EGM_CACHE[key]
    L = _lib.lib()
    stream = stream or torch.cuda.current_stream()
    sp = ctypes.c_void_p(stream.cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def run(cfg):
        _lib.check(L.phs_egm_contract_bf16x3_cfg(T, n_e, T_pad, E_pad, K_pad, p(vh), p(vl), p(mh), p(ml), p(out),
                                                 p(work), cfg, sp), "phs_egm_contract_bf16x3_cfg")

    ms = {}
    for cfg in range(L.phs_egm_bf16x3_config_count()):
        run(cfg)
        times = []
        for _ in range(max(1, repeats)):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            run(cfg)
            e1.record(stream)
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        _lib.check(L.phs_egm_bf16x3_status(p(work), sp), "phs_egm_bf16x3_status")
        ms[cfg] = sorted(times)[len(times) // 2]
    best = min(ms, key=ms.get)
    _EGM_CACHE[key] = (best, ms)
    return best, ms
