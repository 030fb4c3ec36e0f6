"""Launch-shape autotuner of the batched column step (lica_gpu_column_batch_steps_ex_device).

The step kernel runs one CTA per column, persistent over all the steps of a launch.  The
launch shape is the CTA width -- 32, 64, 128 or 256 threads -- which also fixes how many columns
share an SM (8, 4, 2 and 1; a one-warp CTA runs TEMP_EXTP's two phases one after the other).
Results are identical; the speed is not: many short columns favour narrow CTAs and more columns
per SM, a few long ones wide CTAs that finish each column sooner.

``tune(batch)`` times one warm-up step and ``trial_steps`` steps of each shape on a copy of
the batch's device state (the batch itself does not advance), keeps the fastest, and
caches the choice per GPU, kernel generation and batch shape: in memory, and in a JSON file
(``$LICA_TUNE_CACHE``, default ``~/.cache/lica_b200/column_tune.json``) so a later process
on the same GPU model skips the trial.  A choice timed on an earlier generation of the step
kernel is not taken.  ``ColumnBatch.steps(threads=0)`` calls it.
"""
import json
import os
import threading

# (threads, tri_cap); tri_cap, once -1 or 0, has no effect any more
SHAPES = ((32, -1), (64, -1), (128, -1), (256, -1))
# Raised when a change of the step kernel moves the fastest widths.  1: the tridiagonal arrays in
# shared memory or not, 5 columns of 64 threads per SM (its entries name no generation); 2: all
# columns through shared memory of a fixed size, 4 of 64 or 2 of 128 threads per SM.
GENERATION = 2


def _name(shape):
    return f"{shape[0]} threads"


def _shape(entry):
    """A cache entry's shape, or None if its width is none of SHAPES'."""
    try:
        sh = (int(entry["threads"]), int(entry.get("tri_cap", -1)))
    except (KeyError, TypeError, ValueError):
        return None
    return sh if sh[0] in {w for w, _ in SHAPES} and sh[1] in (-1, 0) else None


_lock = threading.Lock()
_memo = {}


def _cache_path():
    return os.environ.get("LICA_TUNE_CACHE",
                          os.path.join(os.path.expanduser("~"), ".cache", "lica_b200", "column_tune.json"))


def _gpu_name(device):
    import torch
    return torch.cuda.get_device_name(device)


def batch_key(batch):
    """Shape of a batch for the cache: column count, total and longest column, and the
    column-length quartiles (the work per CTA and its spread)."""
    import numpy as np
    n = np.asarray(batch.n)
    q = np.percentile(n, [25, 50, 75]).astype(int).tolist()
    return f"ncol={batch.ncol},cells={int(n.sum())},nmax={int(n.max())},q={q[0]}/{q[1]}/{q[2]}"


def cache_key(gpu, batch):
    return f"{gpu}|kernel={GENERATION}|{batch_key(batch)}"


def _load():
    try:
        with open(_cache_path()) as fh:
            return json.load(fh)
    except (OSError, ValueError):
        return {}


def _store(entries):
    path = _cache_path()
    try:
        os.makedirs(os.path.dirname(path), exist_ok=True)
        tmp = path + f".{os.getpid()}.tmp"
        with open(tmp, "w") as fh:
            json.dump(entries, fh, indent=1, sort_keys=True)
        os.replace(tmp, path)
    except OSError:
        pass   # a read-only home: the in-memory cache still holds the choice


def tune(batch, trial_steps=2, force=False):
    """The fastest launch shape for this batch on its GPU: ((threads, tri_cap), {shape name:
    ms per step} of the trial, or None when the choice came from the cache)."""
    import torch
    dev = batch.arrays["w"].device
    key = cache_key(_gpu_name(dev), batch)
    with _lock:
        if not force:
            if key in _memo:
                return _memo[key], None
            disk = _load()
            sh = _shape(disk[key]) if key in disk else None
            if sh is not None:
                _memo[key] = sh
                return sh, None
    times = {}
    for th, cap in SHAPES:
        trial = batch.to(dev)
        trial.steps(1, threads=th, tri_cap=cap)
        torch.cuda.synchronize(dev)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        trial.steps(trial_steps, threads=th, tri_cap=cap)
        b.record()
        torch.cuda.synchronize(dev)
        times[(th, cap)] = a.elapsed_time(b) / trial_steps
        del trial
    best = min(times, key=times.get)
    named = {_name(k): v for k, v in times.items()}
    with _lock:
        _memo[key] = best
        disk = _load()
        disk[key] = {"threads": best[0], "tri_cap": best[1], "ms_per_step": named}
        _store(disk)
    return best, named
