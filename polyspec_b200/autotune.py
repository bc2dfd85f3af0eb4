"""Autotuner of the SHT's pipeline and Legendre tile shapes (no reference
counterpart; the reference's ducc0 picks its own blocking internally).

For each (direction, spin, batch bucket) of a mixed-precision plan the first call
times every candidate -- the mixed pipeline with each allowed number of maps per
CTA of its Legendre kernels, and (for batches of up to 8 maps) the FP64 pipeline
-- with CUDA events, after one untimed run, and keeps the fastest.  Results are
kept per process and in a JSON cache keyed by GPU model, Nside, lmax and the
call's shape, so later processes reuse them; the cache file is $PS_TUNE_CACHE,
default ~/.cache/polyspec_b200/tune.json.

The FP64 pipeline has one candidate: which of its Legendre kernels runs is a rule
on sizes in the library (ps_legendre_f64.cu), not a timing, because their sums
are ordered differently and the same call has to give the same bits in every
process.  An FP64 plan is therefore not timed at all.
"""
import ctypes
import json
import os

import torch

from . import _lib

# tiles to time (as ps_plan_set_tile accepts them; 0: the library's own rule): [pipeline][direction][spin > 0]
TILES = {
    ("mixed", 0, False): (8, 16, 32), ("mixed", 0, True): (4, 8),
    ("mixed", 1, False): (1, 8), ("mixed", 1, True): (1, 4),
    ("fp64", 0, False): (0,), ("fp64", 0, True): (0,),
    ("fp64", 1, False): (0,), ("fp64", 1, True): (0,),
}


def cache_path():
    return os.environ.get("PS_TUNE_CACHE", os.path.join(os.path.expanduser("~"), ".cache", "polyspec_b200",
                                                        "tune.json"))


def _load():
    try:
        with open(cache_path()) as f:
            return json.load(f)
    except Exception:
        return {}


def _save(d):
    try:
        p = cache_path()
        os.makedirs(os.path.dirname(p), exist_ok=True)
        tmp = p + ".tmp%d" % os.getpid()
        with open(tmp, "w") as f:
            json.dump(d, f, indent=1, sort_keys=True)
        os.replace(tmp, p)
    except Exception:
        pass


class Tuner:
    """Per-plan tile and pipeline choices; `handles` maps pipeline name -> plan handle."""

    def __init__(self, nside, lmax, handles, device):
        self.handles = dict(handles)
        try:
            gpu = torch.cuda.get_device_name(device)
        except Exception:
            gpu = "gpu"
        # choices timed with other kernels or among other candidates do not hold ("kernels3"); the
        # pipelines are part of the key
        self.prefix = "%s|kernels3|nside%d|lmax%d|%s" % (gpu, nside, lmax, "+".join(sorted(self.handles)))
        self.choices = {}
        self.picked = {}  # (direction, spin, bucket, table) -> (pipeline, tile)
        self.disk = _load()

    @staticmethod
    def bucket(B):
        if B <= 8:
            return B
        b = 16
        while b < B:
            b *= 2
        return b

    def _set(self, pipeline, direction, spin, tile):
        _lib.call("ps_plan_set_tile", self.handles[pipeline], direction, spin, tile)

    def _candidates(self, direction, spin, B, table):
        """(pipeline, tile) pairs of a call."""
        # the FP64 pipeline only competes for small batches: its workspace is twice the mixed one's (it
        # would win up to about 12 maps of a spin, 16 of spin 0: Nside 256, lmax 511, 0.36 against 0.51 ms for 12)
        pipelines = [pl for pl in self.handles if not (pl == "fp64" and len(self.handles) > 1 and B > 8)]
        return [(pl, tile) for pl in pipelines
                for tile in ((0,) if (table and pl == "mixed") else TILES[(pl, direction, spin > 0)])]

    def select(self, direction, spin, B, run, table=False):
        """Handle to run the transform with (its tile already set); `run(handle)` issues it.
        With `table` the mixed plan streams its Legendre table (ps_plan_build_table): its
        on-the-fly tile shapes do not apply, and the choice is cached under its own key."""
        call = (direction, spin, self.bucket(B), table)
        pick = self.picked.get(call)
        if pick is None:
            pick = self.picked[call] = self._choose(direction, spin, B, run, table)
        pipeline, tile = pick
        self._set(pipeline, direction, spin, tile)
        return self.handles[pipeline]

    def _choose(self, direction, spin, B, run, table):
        cands = self._candidates(direction, spin, B, table)
        if len(cands) == 1:
            return cands[0]
        key = "%s|%s|spin%d|b%d%s" % (self.prefix, ("synthesis", "adjoint")[direction], spin, self.bucket(B),
                                      "|tab" if table else "")
        choice = self.disk.get(key)
        if choice is None or (choice.get("pipeline"), choice.get("tile")) not in cands:
            times = {}
            for pipeline, tile in cands:
                self._set(pipeline, direction, spin, tile)
                h = self.handles[pipeline]
                run(h)
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                run(h)
                e1.record()
                torch.cuda.synchronize()
                times["%s/%d" % (pipeline, tile)] = e0.elapsed_time(e1)
            best = min(times, key=times.get)
            pipeline, tile = best.split("/")
            choice = {"pipeline": pipeline, "tile": int(tile), "ms": times}
            self.disk[key] = choice
            _save(self.disk)
        self.choices[key] = choice
        return choice["pipeline"], choice["tile"]
