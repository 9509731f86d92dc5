"""Launch-shape autotuner for the per-mode kernel.

The kernel's speed depends on where a mode's eight Rodas5 stage vectors live
and on how many modes share an SM (``deb_launch_cfg`` in
``include/discoeb_gb300.h``): in shared memory a mode at nvar 323 takes 44 KB,
with the stage vectors in an L2-resident global array 24 KB, at the price of
an L2 round trip per stage access; registers allow four modes (blocks of four
warps) per SM.  Fewer modes per SM run faster each, more use the FP64 unit
better: which wins depends on the hierarchy sizes, the number of modes and how
unequal they are, so it is
measured, not guessed: :func:`tune` times one launch per candidate shape on
the caller's own workload (CUDA events on the launching stream, after one
untimed launch) and keeps the fastest.  Choices are remembered per (device
name, hierarchy sizes, output count, solver, number of modes within a factor
of two) for the process and, when ``DISCOEB_GB300_TUNE_CACHE`` names a JSON
file, across processes.  A launch of another number of modes does not take
them: the best cap at 256 modes costs 1.8 times the best time at 4096 (below).
"""
from __future__ import annotations

import json
import math
import os

from . import _native

# (stage vectors, modes-per-SM cap); 0 = as many as fit (four by registers).
# One or two modes per SM win where a launch ends on its longest modes: 256 modes
# of nvar 323 take 146 / 155 / 156 ms at 1 / 2 / 4, 4096 take 1051 / 685 / 578.
# "all_global" keeps the whole mode state in L2-resident global memory: at nvar
# 1098 the shared part alone is 72 KB.
CANDIDATES = (("shared", 0), ("shared", 2), ("shared", 1), ("global", 0), ("all_global", 0))

_chosen: dict = {}
_loaded = False

# Choices describe the kernel they were timed with: part of the key, so that a
# file written for another kernel is not taken for this one's.
KERNEL = "4 warps per mode"


def _key(dims: _native.DebDims) -> str:
    import torch

    name = torch.cuda.get_device_name(torch.cuda.current_device())
    return "|".join(str(v) for v in (name, KERNEL, dims.lmaxg, dims.lmaxgp, dims.lmaxr, dims.lmaxnu, dims.nqmax, dims.nout,
                                     dims.return_full, dims.linear_solver))


def _sms() -> int:
    import torch

    return torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count


def mode_class(nmode: int, sms: int) -> int:
    """Launches whose best shape is taken to be the same: up to one mode per
    SM, then by powers of two of modes per SM."""
    return max(0, math.ceil(math.log2(max(nmode, 1) / sms)))


def _count_key(dims: _native.DebDims, nmode: int) -> str:
    return f"{_key(dims)}|modes {mode_class(nmode, _sms())}"


def _cache_path():
    return os.environ.get("DISCOEB_GB300_TUNE_CACHE")


def _load():
    global _loaded
    if _loaded:
        return
    _loaded = True
    path = _cache_path()
    if path and os.path.exists(path):
        try:
            with open(path) as f:
                for k, v in json.load(f).items():
                    _chosen.setdefault(k, (str(v[0]), int(v[1])))
        except (OSError, ValueError, TypeError, IndexError):
            pass


def _store():
    path = _cache_path()
    if not path:
        return
    try:
        os.makedirs(os.path.dirname(os.path.abspath(path)), exist_ok=True)
        with open(path, "w") as f:
            json.dump({k: list(v) for k, v in _chosen.items()}, f, indent=1)
    except OSError:
        pass


def chosen(dims: _native.DebDims, nmode: int | None = None):
    """The remembered launch shape for a launch of ``nmode`` modes of these
    sizes, or None: the one tuned at that number of modes, else the one
    remembered for any number.  Without ``nmode`` the latest choice for these
    sizes, whatever its number of modes."""
    if dims.exec_mode == _native.EXEC_MODES["lane"]:
        return None
    _load()
    if not _chosen:
        return None
    key = _key(dims)
    if nmode is not None:
        return _chosen.get(_count_key(dims, nmode), _chosen.get(key))
    found = [v for k, v in _chosen.items() if k == key or k.startswith(key + "|modes ")]
    return found[-1] if found else None


def remember(dims: _native.DebDims, launch, nmode: int | None = None) -> None:
    """Keep a launch shape for launches of about ``nmode`` modes, or for any
    number of modes that has no choice of its own."""
    _load()
    key = _key(dims) if nmode is None else _count_key(dims, nmode)
    _chosen.pop(key, None)
    _chosen[key] = (str(launch[0]), int(launch[1]))
    _store()


def tune(dims: _native.DebDims, max_modes: int, launch_fn, candidates=CANDIDATES, stream=None):
    """Time ``launch_fn(plan, stream)`` (the launches of one run on ``plan``)
    for every candidate shape on a plan of ``max_modes`` modes; remember (for
    that number of modes) and return ``(best_shape, {shape: ms})``.  Synchronises the device."""
    import torch

    s = stream if stream is not None else torch.cuda.current_stream()
    times = {}
    for cand in candidates:
        try:
            plan = _native.Plan(dims, max_modes, cand)
        except RuntimeError:
            continue   # shape impossible for these sizes (e.g. too large for shared memory)
        info = plan.launch_info()
        shape = (info["stage_vectors"], info["modes_per_sm"])
        if shape in times:
            continue
        launch_fn(plan, s)   # untimed: first-touch of the plan's workspace
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(s)
        launch_fn(plan, s)
        e1.record(s)
        torch.cuda.synchronize()
        times[shape] = e0.elapsed_time(e1)
        del plan
    if not times:
        raise RuntimeError("autotune: no candidate launch shape could be planned")
    best = min(times, key=times.get)
    remember(dims, best, max_modes)
    return best, times
