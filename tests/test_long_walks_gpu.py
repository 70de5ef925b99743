"""Walks far longer than their neighbours: lookups of several values per key
where one key's walk visits the whole table (an absent key in a full one; its
tile of the lookup is then far behind all others, and the call is slow but
answers as any other), and inserts of thousands of values of one key."""
import numpy as np
import pytest
import torch

import warpcore_b200 as wc
from oracle import oracle as o
from tests.wc_helpers import dev, empty_dev, host

pytestmark = pytest.mark.gpu


def device_view(ptr, count):
    """the `count` int32 words at a device pointer as a tensor"""
    class View:
        __cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (ptr, False),
                                    "version": 3}
    return torch.as_tensor(View(), device="cuda")


@pytest.mark.parametrize("kind", ["mv", "mb", "bl"])
def test_absent_key_in_a_full_table(kind):
    slots, real = 1 << 25, 100_003
    keys = o.gen_unique_keys(4, real + 2, 91)
    keys, absent, filler = keys[:real], keys[real], int(keys[real + 1].astype(np.int32))
    values = (np.arange(real) + 1).astype(np.uint32)
    # one value per key: a walk ends where it finds its key
    if kind == "mv":
        t = wc.MultiValueHashTable(slots, key_bytes=4, max_values_per_key=1)
        words = device_view(t.info().slots, 2 * t.capacity)[::2]
    elif kind == "mb":
        t = wc.MultiBucketHashTable(slots, key_bytes=4, bucket_size=1, max_values_per_key=1)
        words = device_view(t.info().keys, t.capacity)
    else:
        t = wc.BucketListHashTable(slots, 2 * real, key_bytes=4, max_values_per_key=1)
        words = device_view(t.info().keys, t.key_capacity)
    t.insert(dev(keys), dev(values))
    words[words == int(np.uint64(t.info().empty_key).astype(np.uint32).astype(np.int32))] = filler
    q = np.concatenate([[absent], keys])  # the long walk is in the first tile
    n = len(q)
    begin, end = (torch.full((n,), -7, dtype=torch.int64, device="cuda") for _ in range(2))
    out, st = empty_dev(real, 4), empty_dev(n, 4)
    assert t.retrieve(dev(q), begin, end, out, status_out=st) == real
    assert np.array_equal(host(end).astype(np.int64), np.arange(n))
    assert np.array_equal(host(begin).astype(np.int64), np.maximum(np.arange(n) - 1, 0))
    assert np.array_equal(host(out).view(np.uint32), values)
    assert np.array_equal(host(st), np.where(np.arange(n) == 0, o.ST_PROBING_LENGTH_EXCEEDED, 0))


@pytest.mark.parametrize("kind", ["mv", "mb1", "mb4"])
@pytest.mark.parametrize("kb,vb,cg", [(4, 4, 8), (8, 8, 8), (4, 8, 1)])
def test_many_values_of_one_key_in_one_batch(kind, kb, vb, cg):
    # a list of more than 128 windows, filled by many warps at once between
    # other keys: every value stored once, one first value per key
    hot, others = 9000 // (8 // cg if cg < 8 else 1), 20_011
    keys = o.gen_unique_keys(kb, others + 1, 107)
    at = np.concatenate([np.full(hot, others), np.arange(others)])
    at = at[np.random.default_rng(17).permutation(len(at))]
    n = len(at)
    vals = (np.arange(n) + 1).astype({4: np.uint32, 8: np.uint64}[vb])
    if kind == "mv":
        t = wc.MultiValueHashTable(2 * n, key_bytes=kb, value_bytes=vb, cg_size=cg)
    else:
        if int(kind[2:]) > cg:
            pytest.skip("buckets are no larger than windows")
        t = wc.MultiBucketHashTable(2 * n, key_bytes=kb, value_bytes=vb, cg_size=cg,
                                    bucket_size=int(kind[2:]))
    st = empty_dev(n, 4)
    t.insert(dev(keys[at]), dev(vals), status_out=st)
    assert t.num_keys() == others + 1
    assert np.count_nonzero(host(st) == o.ST_NONE) == others + 1
    assert np.count_nonzero(host(st) == o.ST_DUPLICATE_KEY) == hot - 1
    begin, end = (torch.zeros(others + 1, dtype=torch.int64, device="cuda") for _ in range(2))
    out = empty_dev(n, vb)
    assert t.retrieve(dev(keys), begin, end, out) == n
    b, e, got = (host(x).astype(np.int64) for x in (begin, end, out))
    owner = np.repeat(np.arange(others + 1), e - b)
    order = np.argsort(got)
    assert np.array_equal(got[order], np.arange(n) + 1)
    assert np.array_equal(owner[order], at)
