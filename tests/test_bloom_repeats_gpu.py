"""Inserts into Bloom filters of keys that are there already: a warp that finds
some reads each block before it sends an OR."""
import numpy as np
import pytest
import torch

import warpcore_b200 as wc
from oracle import oracle as o
from tests.wc_helpers import copy_device_words, dev

pytestmark = pytest.mark.gpu


def stream(kind, n):
    distinct = n // 3
    keys = o.gen_unique_keys(8, distinct, 83)
    rng = np.random.default_rng(7)
    if kind == "zipf":
        return keys[o.gen_zipf_ranks(distinct, 1.1, n, 85).astype(np.int64) - 1]
    if kind == "again":  # every key once, then all of them twice more
        return np.concatenate([keys, keys[::-1], keys])
    if kind == "one":
        return np.full(n, keys[0])
    # distinct keys, long enough that no warp looks any more, then few
    return np.concatenate([keys, keys[rng.integers(0, 5, n - distinct)]])


@pytest.mark.parametrize("kind", ["zipf", "again", "one", "late"])
@pytest.mark.parametrize("sb,cg", [(4, 4), (4, 8), (8, 8), (4, 32), (8, 16)])
@pytest.mark.parametrize("region", [0, 1 << 20])
def test_words_of_repeated_keys(kind, sb, cg, region):
    # every word as by the oracle: one pass and passes over regions, a last
    # block that wraps, two calls so that the second finds all its keys
    num_bits = 8 * sb * (cg * ((5 << 19) // (cg * sb)) + cg // 2)
    keys = stream(kind, 3_000_017)
    prev = wc.set_region_bytes(region)
    try:
        f = wc.BloomFilter(num_bits, 6, key_bytes=8, slot_bytes=sb, cg_size=cg)
        r = o.Bloom(num_bits, 6, key_bytes=8, slot_bytes=sb, cg=cg)
        r.insert(np.unique(keys))
        for _ in range(2):
            f.insert(dev(keys))
            inf = f.info()
            assert np.array_equal(copy_device_words(inf.words, inf.num_slots, sb), r.words())
    finally:
        wc.set_region_bytes(prev)


@pytest.mark.parametrize("sb,cg", [(4, 4), (4, 8), (8, 8), (8, 16)])
@pytest.mark.parametrize("region", [0, 8 << 20])
def test_one_key_many_times_is_not_slow(sb, cg, region):
    # 2^22 copies of one key against 2^22 distinct keys in 32 MiB, device
    # time (15 to 35 times as long with an OR sent for every copy)
    n = 1 << 22
    distinct = torch.empty(n, dtype=torch.int64, device="cuda")
    wc.gen_unique(distinct, 87)
    one = distinct[:1].expand(n).contiguous()
    prev = wc.set_region_bytes(region)
    try:
        f = wc.BloomFilter(1 << 28, 6, key_bytes=8, slot_bytes=sb, cg_size=cg)
        times = []
        for keys in (distinct, one):
            ms = []
            for _ in range(4):
                f.init()
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record()
                f.insert(keys)
                b.record()
                b.synchronize()
                ms.append(a.elapsed_time(b))
            times.append(min(ms[1:]))
    finally:
        wc.set_region_bytes(prev)
    assert times[1] < 6 * times[0], times
