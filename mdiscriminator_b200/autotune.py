"""Autotuner: times the kernels' run-time knobs on this GPU and writes the
table mdiscriminator_b200 loads at import (tuning.json).

Keys: element layout (4-byte values / 8-byte records), class bound (the
smallest power of two >= m) and a range of ceil(log2 n).  Knobs:

* plain path: count and scatter as two kernels against one cooperative
  kernel (`plain_two_kernel`), CTAs per SM of the chunk grid
  (`plain_ctas_per_sm`), the tile geometry (`tile_bytes`: 64 or 32 bytes of
  a tile per thread, `tile_threads`: 256 or 512 threads; two-kernel path) and,
  for the one-kernel path, the share of every chunk drained by ticket
  (`pool_pct`);
* segmented path: tiles per run of a large segment (`run_tiles`),
  small-segment groups per work item (`group_batch`) and whether segments of
  two tiles are read once by the medium-segment kernel (`mid_tiles`).

The reference picked its block shapes by recompiling with -D macros and
timing them (cuda_code/run.py:12-96); here the choice is made at run time.

Usage (on the GPU):  python -m mdiscriminator_b200.autotune [--out PATH] [--quick]
"""
from __future__ import annotations

import argparse
import itertools
import json
import math
import os
import sys
import time

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
if os.path.dirname(HERE) not in sys.path:
    sys.path.insert(0, os.path.dirname(HERE))

import mdiscriminator_b200 as mdx  # noqa: E402

# n buckets: (timed n, ceil(log2 n) range the winner is installed for); the longest
# arrays of 8-byte records have half the count (see timed_count).  Where a grid has few
# tiles a CTA the geometry that wins changes from one power of two to the next, so
# those have a bucket each, timed at three quarters of their range.
BUCKETS = [(1 << 17, (0, 18)), (3 << 18, (19, 20)), (3 << 19, (21, 21)), (3 << 20, (22, 22)),
           (3 << 21, (23, 23)), (3 << 22, (24, 24)), (3 << 23, (25, 25)), (1 << 28, (26, 33))]

# plain-path candidates: (plain_two_kernel, plain_ctas_per_sm, pool_pct, tile_bytes,
# tile_threads).  The one-kernel form (plain_two_kernel = 0) and tiles of 32 bytes per
# thread are not among them: with the present tile steps they were behind at every
# size but for ties.  Inputs of a few tiles take one launch of their own whatever is
# picked here.
PLAIN_CANDIDATES = [(1, 0, 0, 64, 256), (1, 3, 0, 64, 256), (1, 2, 0, 64, 256),
                    (1, 0, 0, 64, 512), (1, 1, 0, 64, 512)]


PLAIN_KNOBS = ("plain_ctas_per_sm", "plain_two_kernel", "pool_pct", "tile_bytes", "tile_threads")


def timed_count(elem, n, bucket):
    """Elements that a bucket is timed at, which lie in it: n, or for 8-byte records in
    the last one half as many (the same bytes)."""
    return n // 2 if elem == mdx.ELEM_REC8 and bucket == BUCKETS[-1][1] else n


def tie(ms):
    """What a candidate has to be below of the best one before it: replays of a few
    microseconds come in steps of two, those of a tenth of a millisecond and more are
    told apart to 1 %."""
    return 0.96 if ms < 0.1 else 0.99


def timeit(graph, torch, reps=9):
    """Median time of one of ten replays of a captured call (no host time between
    its launches)."""
    for _ in range(10):
        graph.launch()
    torch.cuda.synchronize()
    ts = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            graph.launch()
        b.record()
        torch.cuda.synchronize()
        ts.append(a.elapsed_time(b) / 10)
    graph.close()
    return float(np.median(ts))


def lognormal_offsets(n_target, seed):
    rng = np.random.default_rng(seed)
    lengths = []
    total = 0
    while total < n_target:
        L = int(np.clip(np.rint(rng.lognormal(math.log(1024), 1.5)), 1, 1 << 22))
        L = min(L, n_target - total)
        lengths.append(L)
        total += L
    return np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--out", default=mdx.TUNING_PATH)
    ap.add_argument("--quick", action="store_true", help="fewer candidates and sizes")
    ap.add_argument("--elem", choices=("u32", "rec8"), help="this layout only; the table at --out "
                    "keeps its other entries")
    ap.add_argument("--up-to", type=int, default=33, help="buckets up to this log2 n only, likewise")
    ap.add_argument("--plain", action="store_true", help="the plain path's knobs only, likewise")
    args = ap.parse_args(argv)
    kept = {"entries": [], "timings": [], "runs": []}
    if args.elem or args.plain or args.up_to < 33:
        with open(args.out) as f:
            kept = json.load(f)
    import torch
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(1)
    entries = []
    bounds = [2, 4, 8, 16] if args.quick else [2, 4, 8, 16, 32, 64]
    buckets = [b for b in (BUCKETS[1:] if args.quick else BUCKETS) if b[1][1] <= args.up_to]
    t0 = time.time()
    for elem in (mdx.ELEM_U32, mdx.ELEM_REC8):
        ename = "u32" if elem == mdx.ELEM_U32 else "rec8"
        if args.elem not in (None, ename):
            continue
        dtype = torch.int32 if elem == mdx.ELEM_U32 else torch.int64
        for n0, (lo, hi) in buckets:
            n = timed_count(elem, n0, (lo, hi))
            d = torch.randint(0, 1 << 31, (n,), device=dev, dtype=torch.int64, generator=g).to(dtype)
            out = torch.empty_like(d)
            ws = mdx.new_workspace(mdx.workspace_size(n, elem, 64), dev)
            warm = torch.empty(64, dtype=torch.uint32, device=dev)
            for _ in range(200):  # the first candidate is timed on a GPU at speed too
                mdx.partition(d, ("mask", 64), out=out, sizes=warm, ws=ws)
            for M in bounds:
                sizes = torch.empty(M, dtype=torch.uint32, device=dev)
                best = None
                for two, k, pool, tb, tt in PLAIN_CANDIDATES:
                    mdx.set_tuning(elem, M, lo, hi, plain_ctas_per_sm=k, plain_two_kernel=two,
                                   pool_pct=pool, tile_bytes=tb, tile_threads=tt)
                    ms = timeit(mdx.capture_partition(d, ("mask", M), out, sizes, ws=ws), torch)
                    if ws.error() != mdx.MDX_OK:
                        raise SystemExit(f"device error while tuning {ename} m={M}")
                    if best is None or ms < tie(best[0]) * best[0]:  # ties stay with the first
                        best = (ms, k, two, pool, tb, tt)
                entries.append({"elem": ename, "m": M, "log2_n": [lo, hi], "path": "plain",
                                "plain_ctas_per_sm": best[1], "plain_two_kernel": best[2],
                                "pool_pct": best[3], "tile_bytes": best[4],
                                "tile_threads": best[5], "ms": best[0]})
                mdx.set_tuning(elem, M, lo, hi, plain_ctas_per_sm=best[1],
                               plain_two_kernel=best[2], pool_pct=best[3], tile_bytes=best[4],
                               tile_threads=best[5])
            del d, out, ws
        seg_bounds = [2, 4, 8, 16]
        for n0, (lo, hi) in [] if args.plain else buckets:
            n_target = min(timed_count(elem, n0, (lo, hi)), 1 << 27)
            offs = lognormal_offsets(n_target, 3)
            n = int(offs[-1])
            S = len(offs) - 1
            d = torch.randint(0, 1 << 31, (n,), device=dev, dtype=torch.int64, generator=g).to(dtype)
            out = torch.empty_like(d)
            do = torch.from_numpy(offs).to(dev)
            ws = mdx.new_workspace(mdx.segmented_workspace_size(n, S, elem, 16), dev)
            cands = list(itertools.product((2, 4, 8, 16), (2, 4, 8, 16)))
            if args.quick:
                cands = list(itertools.product((4, 8, 16), (8,)))
            for M in seg_bounds:
                ss = torch.empty((S, M), dtype=torch.uint32, device=dev)
                pe = next(e for e in entries
                          if e["elem"] == ename and e["m"] == M and e["path"] == "plain"
                          and e["log2_n"] == [lo, hi])
                plain_k, plain_two, pool = pe["plain_ctas_per_sm"], pe["plain_two_kernel"], pe["pool_pct"]
                tb, tt = pe["tile_bytes"], pe["tile_threads"]
                best = None
                # (run_tiles, group_batch) without medium segments, then the
                # winner with the medium-segment kernel on
                for cand in [(rt, gb, 1) for rt, gb in cands] + [None]:
                    rt, gb, mid = cand if cand is not None else (best[1], best[2], 2)
                    mdx.set_tuning(elem, M, lo, hi, plain_ctas_per_sm=plain_k,
                                   plain_two_kernel=plain_two, pool_pct=pool, tile_bytes=tb,
                                   tile_threads=tt, run_tiles=rt, group_batch=gb, mid_tiles=mid)
                    ms = timeit(mdx.capture_partition_segmented(d, do, ("mask", M), out, ss, ws=ws),
                                torch)
                    if best is None or ms < 0.98 * best[0]:
                        best = (ms, rt, gb, mid)
                entries.append({"elem": ename, "m": M, "log2_n": [lo, hi], "path": "segmented",
                                "plain_ctas_per_sm": plain_k, "plain_two_kernel": plain_two,
                                "pool_pct": pool, "tile_bytes": tb, "tile_threads": tt,
                                "run_tiles": best[1],
                                "group_batch": best[2], "mid_tiles": best[3], "ms": best[0]})
                mdx.set_tuning(elem, M, lo, hi, plain_ctas_per_sm=plain_k,
                               plain_two_kernel=plain_two, pool_pct=pool, tile_bytes=tb,
                               tile_threads=tt, run_tiles=best[1], group_batch=best[2],
                               mid_tiles=best[3])
            del d, out, ws
    # one entry per key: the segmented entry (it carries the plain knob too)
    def key_of(e):
        return e["elem"], e["m"], tuple(e["log2_n"])

    merged = {key_of(e): e for e in kept["entries"]}
    for e in entries:  # a key's segmented entry comes after its plain one
        old = merged.get(key_of(e), e)
        merged[key_of(e)] = {**old, **{k: e[k] for k in PLAIN_KNOBS}} \
            if args.plain and old["path"] == "segmented" else e
    tuned = {(key_of(e), e["path"]) for e in entries}
    table = {"device": torch.cuda.get_device_name(0),
             "runs": kept["runs"] + [{"elem": args.elem or "all",
                                      "path": "plain" if args.plain else "all",
                                      "up_to_log2_n": args.up_to,
                                      "seconds": round(time.time() - t0, 1)}],
             "entries": list(merged.values()),
             "timings": [e for e in kept["timings"] if (key_of(e), e["path"]) not in tuned] + entries}
    with open(args.out, "w") as f:
        json.dump(table, f, indent=1)
    print(f"wrote {len(merged)} entries to {args.out} in {time.time() - t0:.0f} s")


if __name__ == "__main__":
    main()
