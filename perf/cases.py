"""The workloads the library's performance is judged by: one pass of each public
entry point over the sizes, bucket counts, element widths and key distributions
that its users run it at.

Every output is whole numbers (permuted keys and values, offsets, counts).
"""
from __future__ import annotations

import math

import torch

import gpumultisplit_gb300 as gms
from gpumultisplit_gb300 import datagen

LARGEST = 1 << 28


def listed():
    return [
        # A partition step inside a larger GPU program (a join's build side, a
        # work-queue split): a few thousand pairs, the caller needs the bucket
        # bounds on the host.  Latency and launches decide.
        {"name": "pairs_b32_10k", "op": "multisplit", "n": 10007, "buckets": 32, "ident": "delta", "pairs": True,
         "dist": "uniform", "offsets": True},
        # The reference's CPU-runnable case: 2^20 keys by their top three bits.
        {"name": "keys_b8_1m", "op": "multisplit", "n": 1 << 20, "buckets": 8, "ident": "bits", "shift": 29,
         "pairs": False, "dist": "uniform", "offsets": False},
        # The headline: 2^28 pairs into 256 equal ranges.
        {"name": "pairs_b256_256m", "op": "multisplit", "n": LARGEST, "buckets": 256, "ident": "delta",
         "pairs": True, "dist": "uniform", "offsets": False},
        # Range partitioning by sampled splitters (sample sort, shuffles), a
        # size that is no multiple of any tile, bounds returned.
        {"name": "pairs_b32_range_33m", "op": "multisplit", "n": (1 << 25) + 35, "buckets": 32, "ident": "range",
         "pairs": True, "dist": "uniform", "offsets": True},
        # key / delta (the reference's own functor) into a bucket count that is
        # no power of two, on skewed keys.
        {"name": "keys_b100_div_zipf_12m", "op": "multisplit", "n": 12345679, "buckets": 100, "ident": "div",
         "pairs": False, "dist": "zipf", "offsets": False},
        # The reference's headline sort: 7-bit digits, key-value, 2^27 pairs.
        {"name": "sort7_pairs_128m", "op": "sort", "n": 1 << 27, "digit_bits": 7, "pairs": True, "dist": "uniform"},
        # A mid-sized sort of keys alone: five launches' worth of work per pass.
        {"name": "sort8_keys_1m", "op": "sort", "n": 1000003, "digit_bits": 8, "pairs": False, "dist": "uniform"},
        # Stream compaction by a predicate, the count returned to the host.
        {"name": "compact_pairs_128m", "op": "compaction", "n": 1 << 27, "pairs": True, "dist": "uniform"},
        # Even-width histogram of samples, the reference's second tool.
        {"name": "hist_even256_100m", "op": "histogram", "n": 100000007, "buckets": 256, "form": "even",
         "dist": "uniform"},
        # 64-bit keys with 64-bit payloads (pointers, row ids).
        {"name": "wide64_pairs_b256_33m", "op": "wide", "n": (1 << 25) + 77, "buckets": 256, "ident": "delta",
         "key_bytes": 8, "value_bytes": 8, "offsets": False},
        # More than 256 partitions by sampled splitters (a shuffle's fan-out).
        {"name": "pairs_b4096_range_16m", "op": "multisplit", "n": (1 << 24) + 3, "buckets": 4096, "ident": "range",
         "pairs": True, "dist": "uniform", "offsets": False},
        # Many uneven multisplits as one plan: delta and range identifiers, 2
        # to 256 buckets, segments from a handful of keys to a million.
        {"name": "batch_512_segments", "op": "batch", "segments": 512, "lo": 16, "hi": 1 << 20, "layout": 7},
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi]: any integer, now and then a power of two."""
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))
    n = max(lo, min(hi, n))
    if rng.random() < 0.25:
        n = max(lo, min(hi, 1 << (n.bit_length() - 1)))
    return n


def draw(rng):
    op = rng.choice(["multisplit", "multisplit", "multisplit", "multisplit", "big", "sort", "sort", "sort_wide",
                     "compaction", "histogram", "wide", "batch"])
    dist = rng.choice(["uniform", "uniform", "zipf", "and4"])
    pairs = rng.random() < 0.6
    if op == "multisplit":
        ident = rng.choice(["delta", "delta", "range", "div", "bits", "even_float"])
        # powers of two (the reference's counts) as often as any count
        buckets = 1 << rng.randint(1, 8) if ident == "bits" or rng.random() < 0.5 else rng.randint(2, 256)
        case = {"op": op, "n": _size(rng, 4096, LARGEST), "buckets": buckets, "ident": ident, "pairs": pairs,
                "dist": dist, "offsets": rng.random() < 0.4}
        if ident == "bits":
            case["shift"] = rng.choice([0, 32 - (buckets.bit_length() - 1)])
        return case
    if op == "big":
        ident = rng.choice(["delta", "range"])
        return {"op": "multisplit", "n": _size(rng, 65536, 1 << 26), "ident": ident, "pairs": pairs, "dist": dist,
                "buckets": _size(rng, 257, 8192 if ident == "range" else 65536), "offsets": rng.random() < 0.25}
    if op == "sort":
        return {"op": op, "n": _size(rng, 4096, 1 << 26), "digit_bits": rng.choice([4, 5, 6, 7, 7, 8, 8]),
                "pairs": pairs, "dist": dist}
    if op == "sort_wide":
        kb, vb = rng.choice([(8, 0), (8, 4), (8, 8), (4, 8)])
        return {"op": op, "n": _size(rng, 4096, 1 << 25), "key_bytes": kb, "value_bytes": vb,
                "digit_bits": rng.choice([7, 8])}
    if op == "compaction":
        return {"op": op, "n": _size(rng, 4096, 1 << 27), "pairs": pairs, "dist": dist}
    if op == "histogram":
        form = rng.choice(["even", "range", "delta"])
        return {"op": op, "n": _size(rng, 65536, LARGEST), "form": form, "dist": dist,
                "buckets": rng.choice([16, 64, 256, rng.randint(2, 256)] + ([1000, 4096] if form == "delta" else []))}
    if op == "wide":
        kb, vb = rng.choice([(8, 0), (8, 4), (8, 8), (4, 8)])
        return {"op": op, "n": _size(rng, 4096, 1 << 26), "buckets": 1 << rng.randint(1, 8),
                "ident": rng.choice(["delta", "bits", "div"]), "key_bytes": kb, "value_bytes": vb,
                "offsets": rng.random() < 0.3}
    return {"op": op, "segments": rng.randint(64, 1024), "lo": rng.choice([16, 1024]),
            "hi": _size(rng, 1 << 14, 1 << 20), "layout": rng.randint(0, 1 << 20)}


# ------------------------------------------------------------------ inputs
def _keys(case, n, seed):
    dist = case.get("dist", "uniform")
    make = {"uniform": datagen.uniform_u32, "zipf": datagen.zipf_u32, "and4": datagen.and4_u32}[dist]
    return make(n, seed, device="cuda")


def _identifier(case, seed, key_bits=32):
    kind, B = case["ident"], case["buckets"]
    width = -(-(1 << key_bits) // B)  # of B equal ranges of the key space
    if kind == "delta":
        return gms.delta_bucket()
    if kind == "div":
        return gms.delta_func(width)
    if kind == "bits":
        return gms.bits_bucket(case.get("shift", 0))
    if kind == "even_float":
        return gms.even_float_bucket(0, B / float(1 << key_bits))
    return gms.range_bucket(datagen.range_splitters(B, seed, device="cuda"))


def _batch_spec(case):
    return datagen.batched_spec(case["segments"], case["layout"], lo=case["lo"], hi=case["hi"])


def prepare(case, seed):
    op = case["op"]
    s = {"case": case}
    if op == "batch":
        sizes, buckets, kinds = _batch_spec(case)
        # one pooled array per role, each segment starting on a 256-byte boundary
        starts, total = [], 0
        for n in sizes.tolist():
            starts.append(total)
            total += (n + 63) // 64 * 64
        s["kin"] = datagen.uniform_u32(total, seed, device="cuda")
        s["vin"] = datagen.index_values(total, device="cuda")
        s["kout"], s["vout"] = torch.zeros_like(s["kin"]), torch.zeros_like(s["vin"])
        splitters = {int(b): datagen.range_splitters(int(b), seed + int(b), device="cuda") for b in set(buckets)}
        segs = []
        for a, n, b, kind in zip(starts, sizes.tolist(), buckets.tolist(), kinds):
            ident = gms.delta_bucket() if kind == "delta" else gms.range_bucket(splitters[b])
            part = slice(a, a + n)
            segs.append(gms.Segment(s["kin"][part], s["kout"][part], n, b, ident, s["vin"][part], s["vout"][part]))
        s["plan"] = gms.BatchedMultisplit(segs)
        return s

    n = case["n"]
    if op in ("wide", "sort_wide"):
        kb, vb = case["key_bytes"], case["value_bytes"]
        s["kin"] = datagen.uniform_u64(n, seed, device="cuda") if kb == 8 else datagen.uniform_u32(n, seed, device="cuda")
        s["vin"] = None
        if vb:
            s["vin"] = torch.arange(n, dtype=torch.int64 if vb == 8 else torch.int32, device="cuda")
        s["vout"] = None if s["vin"] is None else torch.empty_like(s["vin"])
        s["kout"] = torch.empty_like(s["kin"])
        if op == "wide":
            s["ctx"] = gms.multisplit_context(case["buckets"])
            gms.multisplit_wide_allocate(n, s["ctx"], kb, vb)
            s["ident"] = _identifier(case, seed + 1, 8 * kb)
        else:
            s["ctx"] = gms.ms_sort_context()
            gms.multisplit_sort_wide_allocate(n, s["ctx"], kb, vb, digit_bits=case["digit_bits"])
        return s

    s["kin"] = _keys(case, n, seed)
    if op == "histogram":
        B = case["buckets"]
        s["hist"] = torch.zeros(B, dtype=torch.int32, device="cuda")
        if case["form"] == "range":
            s["levels"] = datagen.range_splitters(B, seed + 1, device="cuda")
        return s
    s["kout"] = torch.empty_like(s["kin"])
    if case["pairs"]:
        s["vin"] = datagen.index_values(n, device="cuda")
        s["vout"] = torch.empty_like(s["vin"])
    if op == "multisplit":
        s["ctx"] = gms.multisplit_context(case["buckets"])
        (gms.multisplit_allocate_key_value if case["pairs"] else gms.multisplit_allocate_key_only)(n, s["ctx"])
        s["ident"] = _identifier(case, seed + 1)
    elif op == "sort":
        s["ctx"] = gms.ms_sort_context()
        name = "multisplit_sort_%dbit" % case["digit_bits"]
        getattr(gms, name + ("_allocate_pairs" if case["pairs"] else "_allocate"))(n, s["ctx"])
        s["sort"] = getattr(gms, name + ("_pairs" if case["pairs"] else ""))
    else:  # compaction
        s["ctx"] = gms.compaction_context()
        (gms.compaction_allocate_key_value if case["pairs"] else gms.compaction_allocate_key_only)(n, s["ctx"])
        s["ident"] = gms.mask_bucket(1)
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "batch":
        s["plan"].run()
        return {"keys": s["kout"], "values": s["vout"]}
    n = case["n"]
    if op == "multisplit":
        offs = True if case["offsets"] else None
        if case["pairs"]:
            o = gms.multisplit_key_value(s["kin"], s["vin"], s["kout"], s["vout"], n, s["ctx"], s["ident"], offs)
        else:
            o = gms.multisplit_key_only(s["kin"], s["kout"], n, s["ctx"], s["ident"], offs)
    elif op == "sort":
        o = None
        if case["pairs"]:
            s["sort"](s["kin"], s["kout"], s["vin"], s["vout"], n, s["ctx"])
        else:
            s["sort"](s["kin"], s["kout"], n, s["ctx"])
    elif op == "compaction":
        if case["pairs"]:
            o = gms.compaction_key_value(s["kin"], s["vin"], s["kout"], s["vout"], n, s["ctx"], s["ident"])
        else:
            o = gms.compaction_key_only(s["kin"], s["kout"], n, s["ctx"], s["ident"])
    elif op == "histogram":
        B = case["buckets"]
        s["hist"].zero_()
        if case["form"] == "even":
            gms.histogram_even(s["kin"], n, s["hist"], B, 0, (1 << 32) - 1, B / 2.0**32)
        elif case["form"] == "range":
            gms.histogram_range(s["kin"], n, s["hist"], B, s["levels"])
        else:
            gms.multisplit_histogram(s["kin"], n, s["hist"], B, gms.delta_bucket())
        return {"counts": s["hist"]}
    elif op == "wide":
        o = gms.multisplit_wide(s["kin"], s["kout"], n, s["ctx"], s["ident"], s["vin"], s["vout"],
                                True if case["offsets"] else None)
    else:
        o = None
        gms.multisplit_sort_wide(s["kin"], s["kout"], n, s["ctx"], s["vin"], s["vout"])
    out = {"keys": s["kout"]}
    if s.get("vout") is not None:
        out["values"] = s["vout"]
    if o is not None:
        # one array rather than up to 64 Ki single numbers
        out["bounds"] = torch.tensor(o, dtype=torch.int64)
    return out


def work(case):
    """Every input byte read once and every output byte written once.  The
    arithmetic is a few integer operations a key, far below the bytes' time."""
    op = case["op"]
    if op == "batch":
        sizes, buckets, _ = _batch_spec(case)
        return {"bytes": int(sizes.sum()) * 16, "flops": 0}
    n = case["n"]
    if op == "histogram":
        return {"bytes": 4 * n + 4 * case["buckets"], "flops": 0}
    if op in ("wide", "sort_wide"):
        per = 2 * (case["key_bytes"] + case["value_bytes"])
    else:
        per = 16 if case["pairs"] else 8
    extra = 4 * case["buckets"] if case.get("offsets") else 0
    if case.get("ident") == "range":
        extra += 4 * case["buckets"]
    return {"bytes": per * n + extra, "flops": 0}


def exact(case, seed):
    """None: every output is whole numbers, which have no error to measure."""
    return None
