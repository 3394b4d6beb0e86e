"""The work a user of this package has it do, as cases to time.

Every case is one pass through a public entry point on inputs that the case
and a seed define, with the output buffers and the workspace a long-running
program keeps.  Whole numbers go in and whole numbers come out, so results are
equal bit for bit or wrong.

* ``plain``    ``partition`` of u32 values or 8-byte {key, payload} records;
* ``records``  ``partition_records`` of rows of any multiple of 4 bytes;
* ``columns``  ``partition_columns`` of a u32 key column and its companions;
* ``segments`` ``partition_segmented`` (offsets, one class count);
* ``flags``    ``mdiscr_segm`` (segment lengths in and class sizes out as head
  flags, the reference's interface);
* ``batch``    ``partition_segmented_multi`` (a class count per segment: the
  launch by which the serving loop answers a batch of requests).
"""
import math

import numpy as np
import torch

import mdiscriminator_b200 as mdx

MAX_SEGMENTS = 200_000
SIGMA = 1.5  # of the log-normal segment lengths


def listed():
    return [
        # One short request: a call on a few thousand values, where launches and latency count.
        {"name": "plain_u32_5k_m4", "kind": "plain", "elem": 4, "n": 5_003, "m": 4, "discr": "mod",
         "keys": "uniform", "flags": False, "offset": 0},
        # A million values in four classes: the size the sequential reference is run at.
        {"name": "plain_u32_1m_m4", "kind": "plain", "elem": 4, "n": 1 << 20, "m": 4, "discr": "mod",
         "keys": "uniform", "flags": False, "offset": 0},
        # The benchmark's headline: 2^28 values in eight classes.
        {"name": "plain_u32_256m_m8", "kind": "plain", "elem": 4, "n": 1 << 28, "m": 8,
         "discr": "mask", "keys": "uniform", "flags": False, "offset": 0},
        # A ragged large array, skewed classes, a remainder that is no power of two.
        {"name": "plain_u32_100m_m13", "kind": "plain", "elem": 4, "n": 100_000_007, "m": 13,
         "discr": "mod", "keys": "zipf", "flags": False, "offset": 0},
        # One radix digit of the most classes the plain path takes.
        {"name": "plain_u32_128m_m64", "kind": "plain", "elem": 4, "n": 1 << 27, "m": 64,
         "discr": "mask", "keys": "uniform", "flags": False, "offset": 0},
        # Key and payload pairs, the benchmark's record configuration.
        {"name": "plain_rec8_128m_m16", "kind": "plain", "elem": 8, "n": 1 << 27, "m": 16,
         "discr": "mask", "keys": "uniform", "flags": False, "offset": 0},
        # Pairs already in class order: every tile holds one class.
        {"name": "plain_rec8_40m_m32_sorted", "kind": "plain", "elem": 8, "n": 40_000_003, "m": 32,
         "discr": "mod", "keys": "sorted", "flags": False, "offset": 0},
        # Rows of five words: the reference's array elements at a width with no kernel of its own.
        {"name": "records_20b_30m_m8", "kind": "records", "bytes": 20, "n": 30_000_001, "m": 8,
         "discr": "mask", "keys": "uniform"},
        # A key with a flag, a short and a wide companion: the reference's tuples of arrays.
        {"name": "columns_20m_m6", "kind": "columns", "widths": "1,2,8", "n": 20_000_003, "m": 6,
         "discr": "mod", "keys": "uniform"},
        # About 100,000 uneven segments in one call: the benchmark's batched configuration.
        {"name": "segments_315m_m4", "kind": "segments", "elem": 4, "n": 315_000_000, "median": 1024,
         "m": 4, "discr": "mod", "flags": False},
        # The same kind of batch through the reference's head-flag interface.
        {"name": "flags_100m_m8", "kind": "flags", "elem": 4, "n": 100_000_000, "median": 1024,
         "m": 8, "discr": "mod"},
        # A full batch of the serving loop: requests of very different length and class count.
        {"name": "batch_16m_mixed", "kind": "batch", "elem": 4, "n": 1 << 24, "lo": 1 << 10,
         "hi": 1 << 20, "m": 16},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _discr(rng, m):
    return rng.choice(("mask", "mod")) if m & (m - 1) == 0 else "mod"


def draw(rng):
    kind = rng.choice(("plain", "plain", "plain", "records", "columns", "segments", "flags", "batch"))
    if kind == "plain":
        elem = rng.choice((4, 4, 8))
        m = rng.choice((2, 4, 8, 16, 32, 64, rng.randint(2, 16), rng.randint(17, 64)))
        return {"kind": kind, "elem": elem, "n": _log_uniform(rng, 1 << 10, (1 << 30) // elem),
                "m": m, "discr": _discr(rng, m), "keys": rng.choice(("uniform", "uniform", "zipf", "sorted")),
                "flags": rng.random() < 0.15, "offset": rng.choice((0, 0, 0, 0, 0, 0, 1, 3))}
    if kind == "records":
        size = rng.choice((12, 16, 20, 24, 32, 40, 64))
        m = rng.randint(2, 32)
        return {"kind": kind, "bytes": size, "n": _log_uniform(rng, 1 << 12, 600_000_000 // size),
                "m": m, "discr": _discr(rng, m), "keys": rng.choice(("uniform", "zipf"))}
    if kind == "columns":
        m = rng.randint(2, 32)
        widths = [rng.choice((1, 2, 4, 8)) for _ in range(rng.randint(1, 4))]
        return {"kind": kind, "widths": ",".join(map(str, widths)), "n": _log_uniform(rng, 1 << 12, 20_000_000),
                "m": m, "discr": _discr(rng, m), "keys": rng.choice(("uniform", "zipf"))}
    if kind == "batch":
        hi = _log_uniform(rng, 1 << 12, 1 << 20)
        return {"kind": kind, "elem": 4, "n": _log_uniform(rng, 1 << 14, 1 << 24), "lo": 1 << 10,
                "hi": hi, "m": rng.choice((4, 8, 16))}
    median = _log_uniform(rng, 32, 1 << 14)
    top = 100_000_000 if kind == "flags" else 300_000_000
    m = rng.randint(2, 16)
    case = {"kind": kind, "elem": rng.choice((4, 4, 8)), "median": median, "m": m, "discr": _discr(rng, m)}
    case["n"] = _log_uniform(rng, 1 << 14, min(top // (case["elem"] // 4), MAX_SEGMENTS * median))
    if kind == "segments":
        case["flags"] = rng.random() < 0.15
    return case


def _keys(n, m, keys, gen):
    """n u32 keys (as int32): uniform, with Zipf(1.1)-distributed classes, or in class order."""
    x = torch.randint(0, 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=gen)
    if keys == "uniform":
        return x
    if keys == "sorted":
        cls = torch.sort((x % m).to(torch.uint8))[0].to(torch.int32)
    else:
        p = torch.arange(1, m + 1, dtype=torch.float64) ** -1.1
        cdf = torch.cumsum(p / p.sum(), 0)[:-1].to("cuda", torch.float32)
        u = torch.rand(n, device="cuda", generator=gen)
        cls = torch.bucketize(u, cdf, right=True, out_int32=True)
    return (x >> 6) // m * m + cls  # key % m is the class, keys stay below 2^31


def _values(n, elem, m, keys, gen):
    k = _keys(n, m, keys, gen)
    if elem == 4:
        return k
    rec = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    rec[:, 0] = k
    rec[:, 1] = torch.arange(n, dtype=torch.int32, device="cuda")
    return rec.view(torch.int64).reshape(n)


def _segments(case):
    """The number of segments of a case, from their mean length."""
    if case["kind"] == "batch":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    else:
        mean = case["median"] * math.exp(SIGMA * SIGMA / 2)
    return max(1, int(case["n"] / mean))


def _lengths(case, seed):
    """Segment lengths adding up to n: log-normal, or log-uniform for a batch of requests."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        x = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), _segments(case)))
    else:
        x = rng.lognormal(math.log(case["median"]), SIGMA, _segments(case))
    ends = np.cumsum(x)
    ends = np.rint(ends * (case["n"] / ends[-1])).astype(np.int64)
    lengths = np.diff(ends, prepend=0)
    return lengths[lengths > 0] if case["kind"] == "flags" else lengths  # head flags know no empty segment


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, m, kind = case["n"], case["m"], case["kind"]
    s = {"kind": kind, "m": m, "discr": (case.get("discr", "mod"), m)}
    if kind == "records":
        size = case["bytes"]
        rows = torch.randint(-(1 << 31), 1 << 31, (n, size // 4), dtype=torch.int32, device="cuda", generator=gen)
        rows[:, 0] = _keys(n, m, case["keys"], gen)
        s.update(x=rows, size=size, out=torch.empty_like(rows))
        s["ws"] = mdx.new_workspace(mdx.lib().mdx_records_workspace_size(n, size, m))
    elif kind == "columns":
        types = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}
        s["x"] = [_keys(n, m, case["keys"], gen)]
        for w in map(int, case["widths"].split(",")):
            raw = torch.randint(0, 256, (n * w,), dtype=torch.uint8, device="cuda", generator=gen)
            s["x"].append(raw.view(types[w]))
        s["out"] = [torch.empty_like(c) for c in s["x"]]
        s["ws"] = mdx.new_workspace(mdx.lib().mdx_columns_workspace_size(n, m))
    elif kind == "plain":
        off = case["offset"]
        x = torch.empty(n + off, dtype=torch.int32 if case["elem"] == 4 else torch.int64, device="cuda")
        x[off:] = _values(n, case["elem"], m, case["keys"], gen)
        s.update(x=x[off:], out=torch.empty_like(x[off:]))
        s["flags"] = torch.empty(n, dtype=torch.int32, device="cuda") if case["flags"] else False
        elem = mdx.ELEM_U32 if case["elem"] == 4 else mdx.ELEM_REC8
        s["ws"] = mdx.new_workspace(mdx.workspace_size(n, elem, m))
    else:
        lengths = _lengths(case, seed)
        elem = mdx.ELEM_U32 if case["elem"] == 4 else mdx.ELEM_REC8
        s["x"] = _values(n, case["elem"], m, "uniform", gen)
        s["out"] = torch.empty_like(s["x"])
        offsets = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)])).cuda()
        S = lengths.size
        if kind == "flags":
            s["lengths"] = torch.zeros(n, dtype=torch.int32, device="cuda")
            s["lengths"][offsets[:-1]] = torch.from_numpy(lengths.astype(np.int32)).cuda()
            s["new"] = torch.empty(n, dtype=torch.int32, device="cuda")
            s["ws"] = mdx.new_workspace(mdx.lib().mdx_mdiscr_segm_workspace_size(n, elem, m))
        else:
            s["offsets"] = offsets
            s["ws"] = mdx.new_workspace(mdx.segmented_workspace_size(n, S, elem, m))
            s["flags"] = torch.empty(n, dtype=torch.int32, device="cuda") if case.get("flags") else False
            if kind == "batch":
                s["seg_m"] = torch.from_numpy(_classes(S, m, seed)).cuda()
            s["sizes"] = torch.empty((S, m), dtype=torch.int32, device="cuda")
    if "sizes" not in s and kind != "flags":
        s["sizes"] = torch.empty(m, dtype=torch.int32, device="cuda")
    return s


def _classes(S, m, seed):
    """Class counts of a batch's requests: powers of two up to m."""
    choices = np.array([c for c in (2, 4, 8, 16) if c <= m], dtype=np.int32)
    return np.random.default_rng(seed + 1).choice(choices, S)


def run(s):
    kind = s["kind"]
    if kind == "plain":
        return mdx.partition(s["x"], s["discr"], out=s["out"], sizes=s["sizes"], headflags=s["flags"], ws=s["ws"])
    if kind == "records":
        return mdx.partition_records(s["x"], s["size"], s["discr"], out=s["out"], sizes=s["sizes"], ws=s["ws"])
    if kind == "columns":
        return mdx.partition_columns(s["x"], s["discr"], outs=s["out"], sizes=s["sizes"], ws=s["ws"])
    if kind == "segments":
        return mdx.partition_segmented(s["x"], s["offsets"], s["discr"], out=s["out"], seg_sizes=s["sizes"],
                                       headflags=s["flags"], ws=s["ws"])
    if kind == "flags":
        return mdx.mdiscr_segm(s["x"], s["lengths"], s["discr"], d_out=s["out"], d_new_sizes=s["new"], ws=s["ws"])
    return mdx.partition_segmented_multi(s["x"], s["offsets"], s["seg_m"], s["m"], out=s["out"],
                                         seg_sizes=s["sizes"], ws=s["ws"])


def work(case):
    """Every input read once and every output written once."""
    n, m, kind = case["n"], case["m"], case["kind"]
    if kind == "records":
        b = 2 * n * case["bytes"] + 4 * m
    elif kind == "columns":
        b = 2 * n * (4 + sum(map(int, case["widths"].split(",")))) + 4 * m
    elif kind == "plain":
        b = 2 * n * case["elem"] + 4 * m + (4 * n if case["flags"] else 0)
    elif kind == "flags":
        b = 2 * n * case["elem"] + 8 * n
    else:
        S = _segments(case)
        b = 2 * n * case["elem"] + 8 * (S + 1) + 4 * m * S + (4 * n if case.get("flags") else 0)
        b += 4 * S if kind == "batch" else 0
    return {"bytes": b, "flops": 0}


def _class_of(keys, m, discr):
    return keys & (m - 1) if discr == "mask" else keys % m


def exact(case, seed):
    """What ``run`` returns, by a stable sort of (segment, class)."""
    s = prepare(case, seed)
    n, m, kind = case["n"], case["m"], case["kind"]
    s["ws"] = None
    if kind in ("plain", "records", "columns"):
        x = s["x"]
        key = x[0] if kind == "columns" else x[:, 0] if kind == "records" else x
        cls = _class_of(key & 0xFFFFFFFF, m, case["discr"]) if kind == "plain" and case["elem"] == 8 else \
            _class_of(key, m, case["discr"])
        order = torch.sort(cls.to(torch.uint8), stable=True)[1]
        sizes = torch.bincount(cls, minlength=m)
        out = [c[order] for c in x] if kind == "columns" else x[order]
        if kind != "plain" or not case["flags"]:
            return out, sizes
        return out, sizes, _head_flags(sizes.reshape(1, m), n)
    lengths = torch.from_numpy(_lengths(case, seed)).cuda()
    S = lengths.numel()
    seg = torch.repeat_interleave(torch.arange(S, device="cuda"), lengths)
    key = s["x"] & 0xFFFFFFFF if case["elem"] == 8 else s["x"]
    if kind == "batch":
        cls = key % s["seg_m"].to(torch.int64)[seg]
    else:
        cls = _class_of(key, m, case["discr"])
    seg = seg * m + cls
    del cls, key
    sizes = torch.bincount(seg, minlength=S * m).reshape(S, m)
    out = s["x"][torch.sort(seg.to(torch.int32), stable=True)[1]]
    if kind == "flags":
        return out, _head_flags(sizes, n)
    return (out, sizes, _head_flags(sizes, n)) if case.get("flags") else (out, sizes)


def _head_flags(sizes, n):
    """Each non-empty class's size at its first position, zero elsewhere."""
    flat = sizes.reshape(-1)
    starts = torch.cumsum(flat, 0) - flat
    hf = torch.zeros(n, dtype=torch.int64, device="cuda")
    hf[starts[flat > 0]] = flat[flat > 0]
    return hf
