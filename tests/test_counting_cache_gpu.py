"""Counting inserts without per-key statuses (the kernel with one count cache
per SM): counts against numpy at the edges of warps, blocks and waves, for
skewed, distinct and constant streams, into filled tables, with invalid
keys, on full tables, with fingerprints, and where a count wraps."""
import numpy as np
import pytest
import torch

import warpcore_b200 as wc
from oracle import oracle as o
from tests.wc_helpers import dev, host

pytestmark = pytest.mark.gpu

DT = {4: np.uint32, 8: np.uint64}


def counts_of(t, keys, vb):
    out = torch.zeros(len(keys), dtype=torch.int32 if vb == 4 else torch.int64, device="cuda")
    t.retrieve(dev(keys), out)
    return host(out).view(DT[vb]).astype(np.int64)


def stream(kind, distinct, n, rng):
    if kind == "constant":
        return np.zeros(n, dtype=np.int64)
    if kind == "distinct":
        return np.arange(n, dtype=np.int64) % distinct
    return np.minimum((distinct ** rng.random(n)).astype(np.int64), distinct) - 1


@pytest.mark.parametrize("kind", ["skewed", "distinct", "constant"])
@pytest.mark.parametrize("kb,vb,cg", [(4, 4, 4), (4, 4, 1), (4, 4, 16), (8, 8, 4), (8, 8, 8),
                                      (8, 4, 2), (4, 8, 8), (8, 8, 16)])
def test_counts(kind, kb, vb, cg):
    distinct = 50000
    keys = o.gen_unique_keys(kb, distinct, 81)
    rng = np.random.default_rng(7)
    t = wc.CountingHashTable(int(distinct / 0.9), key_bytes=kb, value_bytes=vb, cg_size=cg)
    expect = np.zeros(distinct, dtype=np.int64)
    for n in (1, 31, 33, 1023, 1024, 1025, 148 * 1024 + 1, 1000003):
        at = stream(kind, distinct, n, rng)
        t.insert(dev(keys[at]))
        expect += np.bincount(at, minlength=distinct)
        assert np.array_equal(counts_of(t, keys, vb), expect)
        assert t.size() == np.count_nonzero(expect)
    # (lookups of keys that are not counted yet add key_not_found)
    assert int(t.pop_status()) & ~int(wc.Status.key_not_found()) == int(wc.Status.duplicate_key())


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("n", [5000, 600000])
def test_with_fingerprints(kb, n):
    # n of 600 000 of 1 M slots: fingerprints recomputed after the insert;
    # 5000: written by each claim.  Lookups, erases and a second insert read them.
    distinct = 300000
    keys = o.gen_unique_keys(kb, 2 * distinct, 82)
    rng = np.random.default_rng(8)
    prev = wc.set_fingerprint_policy("always")
    try:
        t = wc.CountingHashTable(distinct, key_bytes=kb)
    finally:
        wc.set_fingerprint_policy(prev)
    assert t.has_fingerprints
    expect = np.zeros(2 * distinct, dtype=np.int64)
    for round_ in range(2):
        at = stream("skewed", distinct, n, rng)
        t.insert(dev(keys[at]))
        expect[:distinct] += np.bincount(at, minlength=distinct)
        assert np.array_equal(counts_of(t, keys, kb), expect)
        gone = np.nonzero(expect)[0][::3]
        t.erase(dev(keys[gone]))
        expect[gone] = 0
        assert np.array_equal(counts_of(t, keys, kb), expect)
        assert t.size() == t.size_scan() == np.count_nonzero(expect)


def test_invalid_keys_and_probing_length():
    keys = o.gen_unique_keys(4, 3000, 83)
    t = wc.CountingHashTable(1000, key_bytes=4)
    t.insert(dev(np.array([0, 0xFFFFFFFF] * 50 + [7], dtype=np.uint32)))
    assert int(t.pop_status()) == int(wc.Status.invalid_key())
    assert t.size() == 1
    big = o.gen_unique_keys(4, t.capacity + 5000, 84)
    t.insert(dev(big), probing_length=4)  # one window each: some find it full
    assert int(t.pop_status()) & int(wc.Status.probing_length_exceeded())
    got = counts_of(t, big, 4)
    assert set(np.unique(got)) <= {0, 1}
    t.init()
    t.insert(dev(np.concatenate([keys] * 3)))
    assert (counts_of(t, keys, 4) == 3).all()


def test_wrapped_count_is_reported():
    t = wc.CountingHashTable(1000, key_bytes=4)
    one = torch.full((1 << 28,), 12345, dtype=torch.int32, device="cuda")
    for _ in range(15):
        t.insert(one)
    assert int(t.peek_status()) & int(wc.Status.index_overflow()) == 0
    assert counts_of(t, np.array([12345], dtype=np.uint32), 4)[0] == 15 << 28
    for _ in range(2):
        t.insert(one)
    assert int(t.pop_status()) & int(wc.Status.index_overflow())


def test_two_threads_with_calls_of_other_sizes():
    # each call asks for shared memory by its number of keys; threads must
    # not lower each other's limit
    import threading
    keys = o.gen_unique_keys(4, 400000, 85)
    tables = [wc.CountingHashTable(800000, key_bytes=4) for _ in range(2)]
    inputs = [dev(keys[:1000]), dev(keys)]
    torch.cuda.synchronize()
    errors = []

    def work(t, x):
        try:
            s = torch.cuda.Stream()
            for _ in range(200):
                t.insert(x, stream=s)
            s.synchronize()
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(tables, inputs)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors
    assert (counts_of(tables[0], keys[:1000], 4) == 200).all()
    assert (counts_of(tables[1], keys, 4) == 200).all()
