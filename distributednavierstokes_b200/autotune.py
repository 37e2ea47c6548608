"""Launch-shape autotuner for the batched ensemble (no counterpart in the
reference).

For a periodic box of side n it times one RK3 step under candidate launch
shapes (dnsb_tuning: lines per CTA of the x-, y- and z-transforms, the per-cell
kernels' block shape) by coordinate descent from the defaults: each field in
turn takes the value of its candidates that makes the step fastest (CUDA events
over `steps` steps after two warm-up steps; the best of `repeats` timings), the
others held.  What is returned names the fields that were changed and no others,
so that the rest keep the library's own rules.  The results do not depend on the
shapes, only the time does.  Choices are cached per device name and box in a JSON
file, for the library build that they were timed with.
"""
import hashlib
import json
import os
import time

import torch

from . import _lib, api

CANDIDATES = {
    "lines_z4": (2, 4, 8, 16),
    "lines_y": (2, 4, 8, 16),
    "lines_x": (2, 4, 8),
    "cell": ((64, 2), (32, 4), (128, 2), (32, 8)),
}
# sides whose z-transform is the kernel with a compile-time split, which takes
# lines_z4 (launch_fftz, csrc/dnsb.cu); every other one takes lines_z
Z4_SIDES = (32, 48, 64, 96)


def candidates(n):
    """CANDIDATES for an n^3 box: the z-transform's field is the one its kernel
    reads."""
    return {("lines_z" if f == "lines_z4" and n not in Z4_SIDES else f): v for f, v in CANDIDATES.items()}


def _build_id():
    """What identifies the library build (a timed choice is its build's)."""
    try:
        with open(_lib.LIBPATH, "rb") as f:
            return hashlib.sha256(f.read()).hexdigest()[:16]
    except OSError:
        return None


def default_cache():
    root = os.environ.get("DNSB_TUNE_CACHE") or os.path.join(
        os.environ.get("XDG_CACHE_HOME") or os.path.join(os.path.expanduser("~"), ".cache"), "dnsb")
    return os.path.join(root, "tuning.json")


def _time_step(n, visc, tuning, steps, repeats, device):
    s = api.setup(n=(n, n, n), visc=visc, device=device, tuning=tuning)
    try:
        u = api.random_field(api.vectorfield(s), s, totalenergy=0.5, kpeak=4.0, seed=1)
        p, q = api.scalarfield(s), api.vectorfield(s)
        dt = 0.5 * api.cfl_timestep(u, s, 0.5)
        for _ in range(2):
            api.step(u, p, q, None, s, dt)
        best = float("inf")
        stream = torch.cuda.current_stream(device)
        for _ in range(repeats):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            for _ in range(steps):
                api.step(u, p, q, None, s, dt)
            b.record(stream)
            torch.cuda.synchronize(device)
            best = min(best, a.elapsed_time(b) / steps)
        return best, s.tuning()
    finally:
        s.close()


def tune(n, visc=1e-3, steps=10, repeats=3, device=None, log=None):
    """Coordinate descent over candidates(n) for an n^3 periodic explicit box;
    returns (tuning dict of the changed fields, ms per step, {candidate: ms})."""
    device = device or torch.device("cuda", torch.cuda.current_device())
    cur = {}
    best_ms, _ = _time_step(n, visc, cur, steps, repeats, device)
    tried = {"default": best_ms}
    for field, values in candidates(n).items():
        for v in values:
            trial = dict(cur)
            if field == "cell":
                trial["cell_bx"], trial["cell_by"] = v
            else:
                trial[field] = v
            ms, _ = _time_step(n, visc, trial, steps, repeats, device)
            tried[f"{field}={v}"] = ms
            if ms < best_ms * 0.99:   # keep a change only if it gains more than 1 %
                best_ms, cur = ms, trial
        if log:
            log(f"n={n}: after {field}: {best_ms:.4f} ms {cur}")
    return cur, best_ms, tried


def tune_sizes(sizes, visc=1e-3, cache=None, device=None, log=None, refresh=False):
    """{n: tuning dict} for every box side in `sizes`, from the cache file
    (keyed by device name and side, of this library build) or measured now and
    stored."""
    device = device or torch.device("cuda", torch.cuda.current_device())
    cache = cache or default_cache()
    name = torch.cuda.get_device_name(device)
    data = {}
    if os.path.exists(cache) and not refresh:
        try:
            with open(cache) as f:
                data = json.load(f)
        except (OSError, ValueError):
            data = {}
    out, report, build = {}, {}, _build_id()
    for n in sorted(set(int(v) for v in sizes)):
        key = f"{name}|periodic|{n}"
        if key in data and not refresh and data[key].get("build") == build:
            out[n] = data[key]["tuning"]
            report[n] = dict(data[key], cached=True)
            continue
        t0 = time.perf_counter()
        eff, ms, tried = tune(n, visc, device=device, log=log)
        data[key] = {"tuning": eff, "ms_per_step": ms, "tried": tried, "build": build,
                     "seconds": time.perf_counter() - t0}
        out[n] = eff
        report[n] = dict(data[key], cached=False)
    try:
        os.makedirs(os.path.dirname(cache), exist_ok=True)
        with open(cache + ".tmp", "w") as f:
            json.dump(data, f, indent=1, sort_keys=True)
        os.replace(cache + ".tmp", cache)
    except OSError:
        pass
    return out, report
