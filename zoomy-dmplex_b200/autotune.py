"""Launch-configuration autotuner.

The knobs are the threads per block of the step kernels, the register caps
(resident blocks per SM) of the register-heavy ones, the tile size
(tile_faces; 0 runs the separate face and gather kernels) and, with tiles,
whether one kernel runs the whole stage (fuse_final).  Each trial runs a few
profiled steps (zsme_set_profiling, one CUDA-event pair per launch) and is
scored by the summed time of all the step's kernels.  The tile size comes
first.  Where a trial ran the whole-stage kernel (no separate face-state
launch), its threads per cell are searched with it and the face, face-state
and gather knobs are left alone, which do not act on it; elsewhere the face
block size and register cap are searched with the tile size (they decide each
other's occupancy), then the face-state kernel's form with its cap.  The other
knobs are set one at a time (coordinate descent).  In the end the result and
the configuration that the handle came with are timed in turn on the steps a
program runs (captured, not profiled), and the handle keeps its own unless the
result is faster.  Results are cached in a JSON file keyed by GPU, model,
mesh size and the version of the knobs.

Tuning advances the solver's state: call it right after set_state and load
the initial state again afterwards (``reset``).  Every configuration gives
the same results bit for bit (tests/test_gpu_autotune.py): the knobs change
scheduling and register allocation, not arithmetic.
"""
from __future__ import annotations

import json
import os
import time

from . import native
from .solver import LAUNCH_KEYS, get_launch, set_launch

# tile_faces: also every size that a new handle may start with (multiples of 32 up to 320)
KNOBS = (("tile_faces", (0, 64, 96, 128, 160, 192, 224, 256, 288, 320, 512)), ("face", (64, 128)), ("face_occ", (1, 2, 3, 4)),
         ("prep_lean", (0, 1, 2, 3, 4)), ("prep", (64, 128)), ("prep_occ", (1, 2, 3, 4, 6, 8)), ("gather", (64, 128)),
         ("finalize", (64, 128)), ("finalize_occ", (1, 2, 3, 4)), ("fuse_final", (0, 1)))
# searched together first without the whole-stage kernel: which face path, its
# block size and its register cap decide each other's worth (the fused kernel's
# shared memory per block is fixed by its tile size, so its occupancy depends on
# all three)
JOINT = ("tile_faces", "face", "face_occ")
# then the face-state kernel's form with its register cap (a split form runs
# more threads per cell with fewer registers each, so the cap worth having
# depends on the form)
JOINT_PREP = ("prep_lean", "prep_occ")
# the whole-stage kernel's threads per cell (prep_lean 0 is 1, 3 is 4)
STAGE_THREADS = (1, 2, 4)
# knobs that do not act on the whole-stage kernel
NOT_STAGE = ("face", "face_occ", "prep", "prep_occ", "gather")
# in the cache key: tunings made with other kernels behind the same knobs are not used
VERSION = 2
DEFAULT_CACHE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "tuned_launch.json")


def _gpu_name():
    try:
        import torch
        return torch.cuda.get_device_name(0)
    except Exception:
        return "unknown"


def cache_key(model, n_cells):
    bucket = 1 << max(0, int(n_cells).bit_length() - 1)   # power-of-two size class
    return "%s|%s|%d|v%d" % (_gpu_name(), model, bucket, VERSION)


def load_cache(path=DEFAULT_CACHE):
    """The cached tunings ({} when the file is missing, unreadable or not a
    JSON object: the tuner then measures afresh and rewrites it)."""
    try:
        with open(path) as f:
            db = json.load(f)
    except (OSError, ValueError):
        return {}
    return db if isinstance(db, dict) else {}


def _measure(solver, cfg, steps):
    """Summed device time (ms) of every kernel over `steps` profiled steps, and
    whether they ran the whole-stage kernel.  A first step is not counted: a
    kernel's first launch in a process loads its code between the events."""
    set_launch(solver.h, cfg)
    for n in (1, steps):
        solver.set_profiling(True)                 # from zero
        solver.step(n)
    prof = solver.read_profile() if hasattr(solver, "read_profile") else _read(solver)
    solver.set_profiling(False)
    return sum(ms for ms, n in prof.values()), prof["prep"][1] == 0


def _keep_faster(solver, start, tuned, repeats=3):
    """The one of two configurations whose steps take less time as a program
    runs them: captured steps, both sides twice in turn, the shortest of each."""
    best = {}
    for name, cfg in (("start", start), ("tuned", tuned), ("tuned", tuned), ("start", start)):
        set_launch(solver.h, cfg)
        solver.step(1)                             # captures the step
        for _ in range(repeats):
            solver.sync(False)
            t0 = time.perf_counter()
            solver.step(8)
            solver.sync(False)
            t = time.perf_counter() - t0
            best[name] = min(t, best.get(name, t))
    return tuned if best["tuned"] < best["start"] else start


def _read(solver):
    import ctypes as ct
    import numpy as np
    k = len(native.KERNEL_KINDS)
    ms = np.zeros(k)
    n = (ct.c_int64 * k)()
    native.check(solver.lib.zsme_read_profile(solver.h, ms.ctypes.data_as(ct.POINTER(ct.c_double)), n))
    return {name: (float(ms[i]), int(n[i])) for i, name in enumerate(native.KERNEL_KINDS)}


last_trace = []   # (knob, value, summed kernel ms) of the last tuning run


def tune(solver, model, n_cells, steps=2, cache=DEFAULT_CACHE, use_cache=True, write_cache=True):
    """Pick and apply the fastest launch configuration; returns it (dict).
    The trials of the run are left in last_trace."""
    global last_trace
    key = cache_key(model, n_cells)
    db = load_cache(cache) if use_cache else {}
    if key in db:
        cfg = db[key]["config"]
        set_launch(solver.h, cfg)
        return cfg
    start = get_launch(solver.h)
    cfg = dict(start)
    _measure(solver, cfg, 1)                       # warm-up
    trace = []
    values = dict(KNOBS)
    best, best_t, stage = {}, None, False

    def trial(knob, change):
        """Times cfg with `change`; the fastest of a search stays in best."""
        nonlocal best, best_t, stage
        t, runs_stage = _measure(solver, dict(cfg, **change), steps)
        trace.append((knob, tuple(change.values()) if len(change) > 1 else change[knob], t))
        if best_t is None or t < best_t:
            best, best_t, stage = change, t, runs_stage
        return runs_stage

    for tf in values["tile_faces"]:                # tile size outermost: the tiles are rebuilt per size
        pairs = [(fb, fo) for fb in values["face"] for fo in values["face_occ"]]
        fb, fo = pairs[0]
        if trial("/".join(JOINT), {"tile_faces": tf, "face": fb, "face_occ": fo}):
            for p in STAGE_THREADS:
                trial("tile_faces/prep_lean", {"tile_faces": tf, "prep_lean": p})
            continue
        for fb, fo in pairs[1:]:
            trial("/".join(JOINT), {"tile_faces": tf, "face": fb, "face_occ": fo})
    # the whole-stage kernel leaves the knobs that do not act on it as the handle had them
    cfg.update({k: v for k, v in best.items() if not (stage and k in NOT_STAGE)})
    if not stage:
        best, best_t = {}, None
        for pl in values["prep_lean"]:
            for po in values["prep_occ"]:
                trial("/".join(JOINT_PREP), {"prep_lean": pl, "prep_occ": po})
        cfg.update(best)
    for knob, vals in KNOBS:
        if knob in JOINT or knob in JOINT_PREP or (stage and knob in NOT_STAGE):
            continue
        best, best_t = {}, None
        for v in vals:
            trial(knob, {knob: v})
        cfg.update(best)
    if cfg != start and hasattr(solver, "sync"):   # a stand-in without it only scores its trials
        cfg = _keep_faster(solver, start, cfg)
    last_trace = trace
    set_launch(solver.h, cfg)
    if write_cache:
        db = load_cache(cache)
        db[key] = {"config": cfg, "trace": trace}
        try:
            with open(cache, "w") as f:
                json.dump(db, f, indent=1, sort_keys=True)
        except OSError:
            pass
    return cfg
