"""Workloads by which this library's speed is measured.

A case is a dict of plain values.  ``prepare(case, seed)`` makes what a
program holds before the calls (tables, keys, output buffers, on the GPU),
``run(state)`` is one pass through the public Python API, ``work(case)``
the bytes that the pass cannot do without, and ``exact(case, seed)`` the
answers by plain torch.  ``listed()`` are the standing cases, ``draw(rng)``
gives more of the same ranges.

A build pass starts from ``init``, as a program does that rebuilds its
table, so a pass can be repeated and always ends in the same answers.  The
keys are hashed (distinct, in random order), so no order of the input helps
a table.
"""
import math

import torch

import warpcore_b200 as wc
from warpcore_b200.datagen import uniform_values, unique_keys, zipf_ranks

DEV = "cuda"


def listed():
    return [
        # one request of a key-value service: refresh a few entries of a
        # resident table and look keys up, 80 % of them present
        {"name": "request32", "kind": "request", "key_bytes": 4, "value_bytes": 4,
         "resident": 500_003, "update": 77, "lookup": 300, "hit": 0.8},
        # a tick of a batched server: many requests of uneven size, each on
        # a table of its own, in one call (30 % of them updates)
        {"name": "batch32", "kind": "batch", "key_bytes": 4, "value_bytes": 4, "requests": 48,
         "resident": 700_001, "most": 1 << 16, "updates": 0.3, "hit": 0.8},
        # a table that stays in L2: build and probe, half of the probes miss
        {"name": "pairs32_l2", "kind": "pairs", "key_bytes": 4, "value_bytes": 4,
         "n": 1 << 20, "load": 0.8, "lookup": 1 << 21, "hit": 0.5},
        # the benchmark's table: 64-bit pairs at load 0.9, far larger than L2
        {"name": "pairs64_large", "kind": "pairs", "key_bytes": 8, "value_bytes": 8,
         "n": 1 << 27, "load": 0.9, "lookup": 1 << 27, "hit": 0.5},
        # deduplication with a set that also drops members, ragged size
        {"name": "set64", "kind": "set", "key_bytes": 8, "n": 15_000_017, "load": 0.9,
         "lookup": 15_000_017, "hit": 0.5, "erase": 0.25},
        # k-mer / word counting: a skewed stream, every key's count read back
        {"name": "count32_zipf", "kind": "count", "key_bytes": 4, "draws": 1 << 27,
         "distinct": 1 << 23, "s": 1.1, "load": 0.85},
        # group-by with 64-bit keys and many groups of a few rows
        {"name": "count64_groups", "kind": "count", "key_bytes": 8, "draws": 3_000_001,
         "distinct": 1_000_003, "s": 0.5, "load": 0.8},
        # the benchmark's filter: 2^32 bits, 16 per key, 64-byte blocks
        {"name": "bloom64_large", "kind": "bloom", "key_bytes": 8, "slot_bytes": 8, "cg": 8,
         "k": 8, "bits": 1 << 32, "n": 1 << 28, "lookup": 1 << 28, "hit": 0.5},
        # a join's pre-filter that stays in L2
        {"name": "bloom32_l2", "kind": "bloom", "key_bytes": 4, "slot_bytes": 4, "cg": 8,
         "k": 6, "bits": 1 << 27, "n": 6_000_011, "lookup": 12_000_017, "hit": 0.3},
        # an index with several values per key, filled in rounds; the three
        # tables that hold such indexes, half or more of the lookups absent
        {"name": "multi_value32", "kind": "mv", "key_bytes": 4, "value_bytes": 4,
         "keys": 1 << 22, "per_key": 4, "load": 0.8, "absent": 1 << 22},
        {"name": "multi_bucket32", "kind": "mb", "key_bytes": 4, "value_bytes": 4,
         "keys": 1 << 22, "per_key": 8, "bucket": 4, "load": 0.8, "absent": 12_000_000},
        {"name": "bucket_list32", "kind": "bl", "key_bytes": 4, "value_bytes": 4,
         "keys": 3_000_000, "per_key": 8, "load": 0.9, "absent": 1_500_001},
    ]


def _log(rng, lo, hi):
    """a whole number in [lo, hi], spread over its logarithm"""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["request", "batch", "pairs", "pairs", "set", "count", "bloom", "mv", "mb",
                       "bl"])
    kb, vb = rng.choice([4, 8]), rng.choice([4, 8])
    if kind == "request":
        return {"kind": kind, "key_bytes": kb, "value_bytes": vb,
                "resident": _log(rng, 100_000, 20_000_000), "update": _log(rng, 20, 65_536),
                "lookup": _log(rng, 64, 262_144), "hit": 0.8}
    if kind == "batch":
        return {"kind": kind, "key_bytes": kb, "value_bytes": kb, "requests": rng.randint(4, 64),
                "resident": _log(rng, 100_000, 900_000), "most": _log(rng, 256, 1 << 17),
                "updates": 0.3, "hit": 0.8}
    if kind == "pairs":
        n = _log(rng, 200_000, 60_000_000)
        return {"kind": kind, "key_bytes": kb, "value_bytes": vb, "n": n,
                "load": rng.choice([0.5, 0.7, 0.8, 0.9, 0.95]),
                "lookup": _log(rng, n // 2, 2 * n), "hit": rng.choice([0.2, 0.5, 0.9])}
    if kind == "set":
        n = _log(rng, 100_000, 60_000_000)
        return {"kind": kind, "key_bytes": kb, "n": n, "load": rng.choice([0.5, 0.8, 0.9]),
                "lookup": _log(rng, n // 2, 2 * n), "hit": rng.choice([0.2, 0.5, 0.9]),
                "erase": rng.choice([0.1, 0.25, 0.5])}
    if kind == "count":
        draws = _log(rng, 200_000, 1 << 27)
        return {"kind": kind, "key_bytes": kb, "draws": draws,
                "distinct": _log(rng, max(1000, draws // 64), max(2000, draws // 2)),
                "s": rng.choice([0.5, 0.8, 1.1, 1.3]), "load": rng.choice([0.7, 0.85])}
    if kind == "bloom":
        n = _log(rng, 200_000, 1 << 27)
        return {"kind": kind, "key_bytes": kb, "slot_bytes": rng.choice([4, 8]),
                "cg": rng.choice([1, 2, 4, 8]), "k": rng.choice([4, 6, 8]), "bits": 16 * n, "n": n,
                "lookup": _log(rng, n // 2, 2 * n), "hit": rng.choice([0.1, 0.5, 0.9])}
    keys = _log(rng, 20_000, 1 << 22)
    case = {"kind": kind, "key_bytes": kb, "value_bytes": vb, "keys": keys,
            "per_key": rng.randint(2, 8), "load": rng.choice([0.6, 0.8]),
            "absent": _log(rng, keys // 4, 3 * keys)}
    if kind == "mb":
        case["bucket"] = rng.choice([1, 2, 4, 8])
    return case


# ---- inputs, by seed alone ----

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _lookups(keys, absent, n, hit, gen):
    """n lookups in random order, a fraction `hit` of them stored keys:
    (the keys looked up, the index of each among `keys`, -1 for an absent one)"""
    nh = int(n * hit)
    at = torch.full((n,), -1, dtype=torch.int64, device=DEV)
    if nh:
        at[:nh] = torch.randint(0, keys.numel(), (nh,), device=DEV, generator=gen)
    at = at[torch.randperm(n, device=DEV, generator=gen)]
    q = absent[:n].clone()
    is_hit = at >= 0
    q[is_hit] = keys[at[is_hit]]
    return q, at


def _batch_sizes(case):
    """keys of each request, spread over the logarithm of [64, most]"""
    n, top = case["requests"], math.log(case["most"] / 64)
    return [int(64 * math.exp(top * ((j * 0.618034) % 1.0))) for j in range(n)]


def _inputs(case, seed):
    gen = _gen(seed)
    kind, kb = case["kind"], case["key_bytes"]
    if kind == "batch":
        n, sizes = case["resident"], _batch_sizes(case)
        tables = []
        for j, size in enumerate(sizes):
            both = unique_keys(kb, 0, n + size, (seed * 64 + j) % (1 << 30), DEV)
            keys, values = both[:n].contiguous(), uniform_values(n, kb, gen, DEV)
            update = j < case["updates"] * len(sizes)
            if update:
                at = torch.randint(0, n // size, (1,), device=DEV, generator=gen) + \
                    torch.arange(size, device=DEV) * (n // size)
                q, new = keys[at].contiguous(), uniform_values(size, kb, gen, DEV)
            else:
                q, at = _lookups(keys, both[n:], size, case["hit"], gen)
                new = None
            tables.append((keys, values, q, at, new))
        return {"tables": tables}
    if kind in ("request", "pairs", "set", "bloom"):
        n = case["resident"] if kind == "request" else case["n"]
        lookup = case["lookup"]
        both = unique_keys(kb, 0, n + lookup, seed, DEV)
        d = {"keys": both[:n].contiguous()}
        d["queries"], d["at"] = _lookups(d["keys"], both[n:], lookup, case["hit"], gen)
        if kind in ("request", "pairs"):
            d["values"] = uniform_values(n, case["value_bytes"], gen, DEV)
        if kind == "request":
            at = torch.randperm(n, device=DEV, generator=gen)[:case["update"]]
            d["update_at"], d["update_keys"] = at, d["keys"][at].contiguous()
            d["update_values"] = uniform_values(case["update"], case["value_bytes"], gen, DEV)
        if kind == "set":
            d["erase_at"] = torch.randperm(n, device=DEV, generator=gen)[:int(n * case["erase"])]
            d["erase"] = d["keys"][d["erase_at"]].contiguous()
        return d
    if kind == "count":
        keys = unique_keys(kb, 0, case["distinct"], seed, DEV)
        ranks = zipf_ranks(case["distinct"], case["s"], case["draws"], gen, DEV)
        return {"keys": keys, "ranks": ranks, "stream": keys[ranks].contiguous()}
    # several values per key, inserted in rounds of one value per key
    nk, per = case["keys"], case["per_key"]
    both = unique_keys(kb, 0, nk + case["absent"], seed, DEV)
    rounds = []
    for _ in range(per):
        order = torch.randperm(nk, device=DEV, generator=gen)
        v = uniform_values(nk, case["value_bytes"], gen, DEV)
        v[v == 0] = 1  # a multi-bucket table's empty value
        rounds.append((order, both[:nk][order].contiguous(), v))
    at = torch.randperm(both.numel(), device=DEV, generator=gen)
    return {"rounds": rounds, "queries": both[at].contiguous(), "at": at}


def _int(nbytes):
    return torch.int32 if nbytes == 4 else torch.int64


def prepare(case, seed):
    d = _inputs(case, seed)
    kind, kb = case["kind"], case["key_bytes"]
    s = {"case": case, "in": d, "table": None}
    if kind == "batch":
        looked_up = sum(q.numel() for _, _, q, _, new in d["tables"] if new is None)
        s["out"] = torch.full((looked_up,), -1, dtype=_int(kb), device=DEV)
        s["batch"] = wc.Batch(case["requests"])
        s["requests"], lo = [], 0
        for keys, values, q, _, new in d.pop("tables"):
            t = wc.SingleValueHashTable(keys.numel(), key_bytes=kb)
            t.insert(keys, values)
            if new is not None:
                s["requests"].append((t, "insert", q, new))
            else:
                s["requests"].append((t, "retrieve", q, s["out"][lo:lo + q.numel()]))
                lo += q.numel()
    elif kind in ("request", "pairs"):
        n = d["keys"].numel()
        load = 0.85 if kind == "request" else case["load"]
        s["table"] = wc.SingleValueHashTable(int(n / load), key_bytes=kb,
                                             value_bytes=case["value_bytes"])
        s["out"] = torch.full((case["lookup"],), -1, dtype=_int(case["value_bytes"]), device=DEV)
        if kind == "request":
            s["status"] = torch.zeros(case["lookup"], dtype=torch.int32, device=DEV)
            s["table"].insert(d["keys"], d["values"])
            del d["keys"], d["values"]
        d.pop("at")
    elif kind == "set":
        s["table"] = wc.HashSet(int(case["n"] / case["load"]), key_bytes=kb)
        s["flags"] = [torch.zeros(case["lookup"], dtype=torch.uint8, device=DEV) for _ in range(2)]
        del d["at"], d["erase_at"]
    elif kind == "count":
        s["table"] = wc.CountingHashTable(int(case["distinct"] / case["load"]), key_bytes=kb,
                                          value_bytes=4)
        s["out"] = torch.zeros(case["distinct"], dtype=torch.int32, device=DEV)
        del d["ranks"]
    elif kind == "bloom":
        s["table"] = wc.BloomFilter(case["bits"], case["k"], key_bytes=kb,
                                    slot_bytes=case["slot_bytes"], cg_size=case["cg"])
        s["flags"] = torch.zeros(case["lookup"], dtype=torch.uint8, device=DEV)
        # a view of the filter's memory: it keeps the filter alive
        s["words"] = s["table"].words_tensor()
        s["words"].of_filter = s["table"]
        del d["at"]
    else:
        nk, per, vb = case["keys"], case["per_key"], case["value_bytes"]
        if kind == "mv":
            s["table"] = wc.MultiValueHashTable(int(nk * per / case["load"]), key_bytes=kb,
                                                value_bytes=vb)
        elif kind == "mb":
            slots = nk * -(-per // case["bucket"])
            s["table"] = wc.MultiBucketHashTable(int(slots / case["load"]), key_bytes=kb,
                                                 value_bytes=vb, bucket_size=case["bucket"])
        else:
            s["table"] = wc.BucketListHashTable(int(nk / case["load"]), 3 * nk * per, key_bytes=kb,
                                                value_bytes=vb)
        nq = d["queries"].numel()
        s["begin"] = torch.zeros(nq, dtype=torch.int64, device=DEV)
        s["end"] = torch.zeros(nq, dtype=torch.int64, device=DEV)
        s["out"] = torch.zeros(nk * per, dtype=_int(vb), device=DEV)
        d["rounds"] = [(k, v) for _, k, v in d["rounds"]]
        del d["at"]
    return s


def run(s):
    case, d, t = s["case"], s["in"], s["table"]
    kind = case["kind"]
    if kind == "request":
        t.insert(d["update_keys"], d["update_values"])
        t.retrieve(d["queries"], s["out"], status_out=s["status"])
        return s["out"], s["status"]
    if kind == "batch":
        s["batch"].run(s["requests"])
        return s["out"]
    t.init()
    if kind == "pairs":
        t.insert(d["keys"], d["values"])
        t.retrieve(d["queries"], s["out"])
        return s["out"]
    if kind == "set":
        t.insert(d["keys"])
        t.retrieve(d["queries"], s["flags"][0])
        t.erase(d["erase"])
        t.retrieve(d["queries"], s["flags"][1])
        return s["flags"][0], s["flags"][1], t.size()
    if kind == "count":
        t.insert(d["stream"])
        t.retrieve(d["keys"], s["out"])
        return s["out"]
    if kind == "bloom":
        t.insert(d["keys"])
        t.retrieve(d["queries"], s["flags"])
        return s["flags"], s["words"]
    for keys, values in d["rounds"]:
        t.insert(keys, values)
    total = t.retrieve(d["queries"], s["begin"], s["end"], s["out"])
    return s["begin"], s["end"], s["out"], total


def work(case):
    """keys, values and lookups read once, answers written once, and the
    stored state written once (and read once by the lookups, at most whole)"""
    kind, kb, vb = case["kind"], case["key_bytes"], case.get("value_bytes", 0)
    if kind == "request":
        n, q = case["update"], case["lookup"]
        return {"bytes": n * 2 * (kb + vb) + q * (2 * (kb + vb) + 4), "flops": 0}
    if kind == "batch":
        return {"bytes": sum(_batch_sizes(case)) * 4 * kb, "flops": 0}
    if kind == "pairs":
        n, q = case["n"], case["lookup"]
        return {"bytes": n * (2 + 1 / case["load"]) * (kb + vb) + q * (kb + vb * case["hit"]),
                "flops": 0}
    if kind == "set":
        n, q = case["n"], case["lookup"]
        return {"bytes": n * kb * (3 + 1 / case["load"] + case["erase"]) + 2 * q * (kb + 1),
                "flops": 0}
    if kind == "count":
        return {"bytes": case["draws"] * kb + case["distinct"] * (2 + 1 / case["load"]) * (kb + 4),
                "flops": 0}
    if kind == "bloom":
        return {"bytes": case["n"] * kb + case["lookup"] * (kb + 1) + 2 * case["bits"] / 8,
                "flops": 0}
    pairs, q = case["keys"] * case["per_key"], case["keys"] + case["absent"]
    return {"bytes": pairs * (2 * (kb + vb) + 2 * vb) + q * (kb + 16), "flops": 0}


def exact(case, seed):
    """the answers of run(), by plain torch; a filter's flags and words have
    no value without its hash function"""
    kind = case["kind"]
    if kind == "bloom":
        return None
    d = _inputs(case, seed)
    if kind == "batch":
        return torch.cat([torch.where(at >= 0, values[at.clamp(min=0)], -1)
                          for _, values, _, at, new in d["tables"] if new is None])
    if kind in ("request", "pairs"):
        values, at = d["values"].clone(), d["at"]
        if kind == "request":
            values[d["update_at"]] = d["update_values"]
        out = torch.where(at >= 0, values[at.clamp(min=0)], torch.full_like(values[:1], -1))
        if kind == "pairs":
            return out
        return out, torch.where(at >= 0, 0, 1 << 5).to(torch.int32)  # Status key_not_found
    if kind == "set":
        gone = torch.zeros(case["n"], dtype=torch.bool, device=DEV)
        gone[d["erase_at"]] = True
        at = d["at"]
        first = at >= 0
        second = first & ~gone[at.clamp(min=0)]
        return first.to(torch.uint8), second.to(torch.uint8), case["n"] - d["erase_at"].numel()
    if kind == "count":
        return torch.bincount(d["ranks"], minlength=case["distinct"]).to(torch.int32)
    nk, per = case["keys"], case["per_key"]
    at = d["at"]
    counts = torch.where(at < nk, per, 0)
    end = torch.cumsum(counts, 0)
    if kind == "bl":
        return end - counts, end, None, nk * per  # its value order is the buckets'
    stored = torch.empty((nk, per), dtype=d["rounds"][0][2].dtype, device=DEV)
    for j, (order, _, v) in enumerate(d["rounds"]):
        stored[order, j] = v
    return end - counts, end, stored[at[at < nk]].reshape(-1), nk * per
