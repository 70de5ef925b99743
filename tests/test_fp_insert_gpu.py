"""Inserts that read fingerprints first, where several lanes hold one key."""
import numpy as np
import pytest
import torch

import warpcore_b200 as wc
from oracle import oracle as o
from tests.wc_helpers import copy_device_words, dev, empty_dev, host

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _fingerprints():
    prev = wc.set_fingerprint_policy("always")
    yield
    wc.set_fingerprint_policy(prev)


def bytes_view(ptr, count):
    class View:
        __cuda_array_interface__ = {"shape": (count,), "typestr": "|u1", "data": (ptr, False),
                                    "version": 3}
    return torch.as_tensor(View(), device="cuda")


@pytest.mark.parametrize("cg", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("kb", [4, 8])
def test_fingerprint_seen_before_its_key(kb, cg):
    # an insert writes the key, then its fingerprint, and another lane may
    # see them the other way round: the slot still reads empty.  Its claim
    # has to decide, or the key takes a second slot.  Here every slot is in
    # that state: the key must go to the first slot of its first window.
    key, val = o.gen_unique_keys(kb, 1, 17), o.gen_uniform(kb, 1, 18)
    plain = wc.SingleValueHashTable(4096, key_bytes=kb, cg_size=cg)
    plain.insert(dev(key), dev(val))
    fps = copy_device_words(plain.info().fingerprints, plain.capacity, 1)
    at = int(np.flatnonzero(fps)[0])
    t = wc.SingleValueHashTable(4096, key_bytes=kb, cg_size=cg)
    bytes_view(t.info().fingerprints, t.capacity).fill_(int(fps[at]))
    st = empty_dev(1, 4)
    t.insert(dev(key), dev(val), status_out=st)
    assert host(st)[0] == o.ST_NONE
    words = copy_device_words(t.info().slots, 2 * t.capacity, kb)
    assert np.array_equal(words, copy_device_words(plain.info().slots, 2 * t.capacity, kb))
    assert t.size() == 1


@pytest.mark.parametrize("cg", [1, 4, 8, 32])
@pytest.mark.parametrize("kb,vb", [(4, 4), (8, 8), (4, 8), (8, 4)])
def test_equal_keys_of_one_call(kb, vb, cg):
    # up to 32 keys in a call: the first of equal keys claims the slot, the
    # last one's value is stored, whether the key is new or not
    rng = np.random.default_rng(3)
    pool = o.gen_unique_keys(kb, 64, 23)
    t = wc.SingleValueHashTable(2000, key_bytes=kb, value_bytes=vb, cg_size=cg)
    stored = {}
    for call in range(60):
        n = int(rng.integers(1, 33))
        at = rng.integers(0, min(len(pool), 1 + call * 2), n)
        vals = rng.integers(1, 2**31, n).astype({4: np.uint32, 8: np.uint64}[vb])
        st = empty_dev(n, 4)
        t.insert(dev(pool[at]), dev(vals), status_out=st)
        want = []
        for k, v in zip(at, vals):
            want.append(o.ST_DUPLICATE_KEY if k in stored else o.ST_NONE)
            stored[k] = v
        assert np.array_equal(host(st), want)
        out = empty_dev(len(stored), vb)
        t.retrieve(dev(pool[list(stored)]), out)
        assert np.array_equal(host(out), np.array(list(stored.values())))
        assert t.size() == len(stored)


@pytest.mark.parametrize("preload", [False, True])
@pytest.mark.parametrize("kb,vb", [(4, 4), (8, 8), (4, 8), (8, 4)])
def test_claims_over_stale_payloads(kb, vb, preload):
    # free slots whose payload is not zero, with and without a load of the
    # slot before its claim (bit 4): every key is stored once
    n = 50_021
    keys, vals = o.gen_unique_keys(kb, n, 25), o.gen_uniform(vb, n, 27)
    at = np.concatenate([np.arange(n), np.arange(0, n, 3)])
    prev = wc.set_fingerprint_ops(0x1F if preload else 0xF)
    try:
        t = wc.SingleValueHashTable(2 * n, key_bytes=kb, value_bytes=vb)
        inf = t.info()
        slots = bytes_view(inf.slots, t.capacity * inf.slot_bytes).view(t.capacity, inf.slot_bytes)
        first = inf.slot_bytes // 2  # the payload follows the key
        slots[::2, first:first + vb] = 7
        for claims in (n, 0):
            st = empty_dev(len(at), 4)
            t.insert(dev(keys[at]), dev(vals[at]), status_out=st)
            assert np.count_nonzero(host(st) == o.ST_NONE) == claims
            assert t.size() == t.size_scan() == n
            out = empty_dev(n, vb)
            t.retrieve(dev(keys), out)
            assert np.array_equal(host(out), vals)
    finally:
        wc.set_fingerprint_ops(prev)


@pytest.mark.parametrize("kind", ["pairs32", "pairs64", "set32", "set64"])
@pytest.mark.parametrize("skew", ["zipf", "runs", "one", "late"])
def test_repeated_keys(kind, skew):
    # equal keys merged or not, by refill: one slot per key, a value that
    # came with it, one status none per new key
    kb = 4 if kind.endswith("32") else 8
    n, distinct = 300_007, 20_011
    keys = o.gen_unique_keys(kb, distinct, 29)
    rng = np.random.default_rng(4)
    if skew == "zipf":
        at = o.gen_zipf_ranks(distinct, 1.2, n, 31).astype(np.int64) - 1
    elif skew == "runs":
        at = np.repeat(np.arange(distinct), 15)[:n]
    elif skew == "one":
        at = np.zeros(n, dtype=np.int64)
    else:  # distinct keys first, then four
        at = np.concatenate([np.arange(distinct), rng.integers(0, 4, n - distinct)])
    n = len(at)
    t = wc.HashSet(3 * distinct, key_bytes=kb) if kind.startswith("set") else \
        wc.SingleValueHashTable(3 * distinct, key_bytes=kb)
    st = empty_dev(n, 4)
    held = len(np.unique(at))
    for call in range(2):
        if kind.startswith("set"):
            t.insert(dev(keys[at]), status_out=st)
        else:  # the value tells the key and the place in the input
            vals = (at * 2**15 % 2**31 + np.arange(n) % 2**15).astype(keys.dtype)
            t.insert(dev(keys[at]), dev(vals), status_out=st)
        got = host(st)
        assert np.count_nonzero(got == o.ST_NONE) == (held if call == 0 else 0)
        assert np.count_nonzero(got == o.ST_DUPLICATE_KEY) == n - (held if call == 0 else 0)
        assert t.size() == t.size_scan() == held
    if not kind.startswith("set"):
        present = np.unique(at)
        out = empty_dev(len(present), kb)
        t.retrieve(dev(keys[present]), out)
        assert np.array_equal(host(out).astype(np.int64) >> 15, present * 2**15 % 2**31 >> 15)


@pytest.mark.parametrize("kind", ["pairs32", "pairs64", "set64"])
def test_one_key_many_times_is_not_slow(kind):
    # 2^22 copies of one key against 2^22 distinct keys, device time (2 to 15
    # times as long with a claim and a store per copy, 0.6 to 2.5 merged)
    kb, n = (4 if kind.endswith("32") else 8), 1 << 22
    t = wc.HashSet(4 * n, key_bytes=kb) if kind == "set64" else \
        wc.SingleValueHashTable(4 * n, key_bytes=kb)
    distinct = torch.empty(n, dtype={4: torch.int32, 8: torch.int64}[kb], device="cuda")
    wc.gen_unique(distinct, 37)
    one = distinct[:1].expand(n).contiguous()
    times = []
    for keys in (distinct, one):
        ms = []
        for _ in range(4):
            t.init()
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            t.insert(keys) if kind == "set64" else t.insert(keys, distinct)
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        times.append(min(ms[1:]))
    assert times[1] < 6 * times[0], times


@pytest.mark.parametrize("kind", ["count32", "count64", "count64_32", "set32"])
def test_rebuild_keeps_fingerprints_of_other_claims(kind):
    # a large insert writes no fingerprints and has them recomputed after; a
    # slot that it reads as empty may be claimed by another stream's insert
    # before it writes, and that one's fingerprint must stay.  Here every
    # empty slot is in that state.
    if kind == "set32":  # (sets rebuild where fingerprints exceed half of L2)
        kb = 4
        cap = torch.cuda.get_device_properties(0).L2_cache_size // 2 + (1 << 20)
        t = wc.HashSet(cap, key_bytes=4)
    else:
        kb, vb = {"count32": (4, 4), "count64": (8, 8), "count64_32": (8, 4)}[kind]
        t = wc.CountingHashTable(1_000_003, key_bytes=kb, value_bytes=vb)
    n = t.capacity // 4
    keys = torch.empty(n, dtype={4: torch.int32, 8: torch.int64}[kb], device="cuda")
    wc.gen_unique(keys, 39)
    fps = bytes_view(t.info().fingerprints, t.capacity)
    fps.fill_(255)
    t.insert(keys)
    assert t.size() == t.size_scan() == n
    assert bool((fps != 0).all())
    assert int((fps != 255).sum()) > n * 9 // 10  # the stored keys' were written
    if kind == "set32":
        out = torch.zeros(n, dtype=torch.uint8, device="cuda")
        t.retrieve(keys, out)
    else:
        out = empty_dev(n, vb)
        t.retrieve(keys, out)
    assert bool((out == 1).all())
