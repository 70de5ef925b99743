"""Counting inserts without statuses of streams whose order works against the
count cache: rare keys first, runs, sorted keys."""
import numpy as np
import pytest
import torch

import warpcore_b200 as wc
from oracle import oracle as o
from tests.wc_helpers import dev, empty_dev, host

pytestmark = pytest.mark.gpu

WARPS = 148 * 32  # of the counting kernel, each with a range of its own


def late(n, distinct, rng):
    # the first 300 keys of each warp's range are distinct, the rest few
    per = -(-(-(-n // WARPS)) // 32) * 32
    i = np.arange(n)
    return np.where(i % per < 300, (i // per * 300 + i % per) % distinct,
                    rng.integers(0, 16, n))


def stream(kind, n, distinct):
    rng = np.random.default_rng(11)
    if kind == "late":
        return late(n, distinct, rng)
    if kind == "runs":
        return np.arange(n) // 13 % distinct
    zipf = o.gen_zipf_ranks(distinct, 0.9, n, 91).astype(np.int64) - 1
    if kind == "sorted":
        return np.sort(zipf)
    # one key, then keys in an order without equal ones nearby
    return np.concatenate([np.zeros(n // 2, dtype=np.int64), np.arange(n - n // 2) % distinct])


@pytest.mark.parametrize("kind", ["late", "runs", "sorted", "one_then_all"])
@pytest.mark.parametrize("kb,vb,cg", [(4, 4, 8), (8, 8, 8), (8, 4, 4), (4, 8, 1)])
def test_counts(kind, kb, vb, cg):
    n, distinct = 3_000_017, 100_003
    keys = o.gen_unique_keys(kb, distinct, 93)
    at = stream(kind, n, distinct)
    t = wc.CountingHashTable(2 * distinct, key_bytes=kb, value_bytes=vb, cg_size=cg)
    counts = np.bincount(at, minlength=distinct)
    present = np.flatnonzero(counts)
    for call in (1, 2):
        t.insert(dev(keys[at]))
        out = empty_dev(len(present), vb)
        t.retrieve(dev(keys[present]), out)
        assert np.array_equal(host(out).astype(np.int64), call * counts[present])
        assert t.size() == t.size_scan() == len(present)
        assert int(t.pop_status()) == o.ST_DUPLICATE_KEY


@pytest.mark.parametrize("kb", [4, 8])
def test_rare_keys_first_is_not_slow(kb):
    # device time against the same keys in random order (16 times as long or
    # more for a warp that leaves the cache out for good)
    n, distinct = 1 << 24, 1 << 20
    rng = np.random.default_rng(12)
    keys = o.gen_unique_keys(kb, distinct, 95)[late(n, distinct, rng)]
    t = wc.CountingHashTable(2 * distinct, key_bytes=kb, value_bytes=4)
    times = []
    for order in (dev(keys), dev(rng.permutation(keys))):
        ms = []
        for _ in range(4):
            t.init()
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            t.insert(order)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        times.append(min(ms[1:]))
    assert times[0] < 8 * times[1], times
