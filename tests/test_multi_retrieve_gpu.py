"""The lookups and inserts of the multi-value, multi-bucket and bucket-list
tables at the edges of their tiles: query counts around a block's threads, a
full tile and a full wave, keys whose values fill many windows, a key with
tens of thousands of values, input counts around warps, queues and waves.
(Two tests are named after notes of the windows found, which an earlier form
of the lookup kept.)"""
import numpy as np
import pytest
import torch

import warpcore_b200 as wc
from oracle import oracle as o
from tests.wc_helpers import dev, empty_dev, host

pytestmark = pytest.mark.gpu

DT = {4: np.uint32, 8: np.uint64}


def make(kind, kb, vb, nkeys, per, load=0.8):
    if kind == "mv":
        return wc.MultiValueHashTable(int(nkeys * per / load), key_bytes=kb, value_bytes=vb)
    if kind == "mb":
        return wc.MultiBucketHashTable(int(nkeys * -(-per // 4) / load), key_bytes=kb,
                                       value_bytes=vb, bucket_size=4)
    return wc.BucketListHashTable(int(nkeys / load), 4 * nkeys * per, key_bytes=kb, value_bytes=vb)


def retrieve(t, queries, total, vb, joined=False):
    n = len(queries)
    off = torch.full((n + 1,), -7, dtype=torch.int64, device="cuda")
    begin, end = off[:n], off[1:]
    if not joined:
        begin = torch.full((n,), -7, dtype=torch.int64, device="cuda")
    out = empty_dev(max(total, 1), vb)
    st = empty_dev(n, 4)
    num = t.retrieve(dev(queries), begin, end, out, status_out=st)
    return num, host(begin).astype(np.int64), host(end).astype(np.int64), host(out)[:num], host(st)


@pytest.mark.parametrize("kind", ["mv", "mb", "bl"])
@pytest.mark.parametrize("kb,vb", [(4, 4), (8, 8), (4, 8), (8, 4)])
def test_tile_edges(kind, kb, vb):
    nkeys, per = 3000, 5
    both = o.gen_unique_keys(kb, 2 * nkeys, 77)
    keys = both[:nkeys]
    rng = np.random.default_rng(5)
    values = rng.integers(1, 2**31, size=(nkeys, per)).astype(DT[vb])
    t = make(kind, kb, vb, nkeys, per)
    for j in range(per):  # one value of each key per round: the order is known
        t.insert(dev(keys), dev(np.ascontiguousarray(values[:, j])))
    # a bucket list is read newest bucket first: buckets of 1, 2, 3 values
    order = [3, 4, 1, 2, 0] if kind == "bl" else range(per)
    for n in (1, 31, 255, 256, 257, 1024, 1025, 2048, 2049, 148 * 6 * 256 + 1,
              148 * 6 * 1024 + 1025, 148 * 6 * 2048 + 2049):
        at = rng.integers(0, 2 * nkeys, size=n)
        hit = at < nkeys
        cnt = np.where(hit, per, 0)
        num, b, e, v, st = retrieve(t, both[at], int(cnt.sum()), vb, joined=n % 2 == 1)
        assert num == cnt.sum()
        assert np.array_equal(e, np.cumsum(cnt))
        assert np.array_equal(b, np.cumsum(cnt) - cnt)
        assert np.array_equal(v.view(DT[vb]), values[at[hit]][:, list(order)].reshape(-1))
        assert np.array_equal(st, np.where(hit, 0, 1 << 5))
        counts = torch.zeros(n, dtype=torch.int64, device="cuda")
        assert t.num_values(dev(both[at]), counts) == num
        assert np.array_equal(host(counts).astype(np.int64), cnt)


@pytest.mark.parametrize("kind", ["mv", "mb"])
@pytest.mark.parametrize("kb", [4, 8])
def test_more_windows_than_notes(kind, kb):
    # 60 values in windows of 8 (or buckets of 4 in such windows): more than
    # the two notes per key that a tile holds, so keys are walked again
    nkeys, per = 2048, 60
    keys = o.gen_unique_keys(kb, nkeys, 78)
    rng = np.random.default_rng(6)
    values = rng.integers(1, 2**31, size=(nkeys, per)).astype(DT[kb])
    t = make(kind, kb, kb, nkeys, per, load=0.9)
    for j in range(per):
        t.insert(dev(keys), dev(np.ascontiguousarray(values[:, j])))
    q = np.concatenate([keys] * 80)  # full tiles, every query present
    num, b, e, v, _ = retrieve(t, q, len(q) * per, kb)
    assert num == len(q) * per
    assert np.array_equal(e, (np.arange(len(q)) + 1) * per)
    assert np.array_equal(v.view(DT[kb]), np.concatenate([values.reshape(-1)] * 80))


def test_key_with_more_values_than_a_note_counts():
    n, extra = 40000, 1000
    keys = o.gen_unique_keys(4, extra + 1, 79)
    t = wc.MultiValueHashTable(int((n + extra) / 0.5), key_bytes=4)
    vals = np.arange(1, n + 1, dtype=np.uint32)
    t.insert(dev(keys[1:]), dev(vals[:extra]))
    t.insert(dev(np.full(n, keys[0], dtype=np.uint32)), dev(vals))
    q = np.concatenate([keys[1:], keys[:1], keys[1:]])
    num, b, e, v, _ = retrieve(t, q, n + 2 * extra, 4)
    assert num == n + 2 * extra
    assert np.array_equal(v[:extra], vals[:extra])
    assert np.array_equal(np.sort(v[extra:extra + n].view(np.uint32)), vals)
    assert np.array_equal(v[extra + n:], vals[:extra])


@pytest.mark.parametrize("kb,vb", [(4, 4), (8, 8), (8, 4)])
@pytest.mark.parametrize("cg", [1, 8, 16, 32])
def test_insert_sizes_and_limits(kb, vb, cg):
    # input counts around a warp, its two prefetch buffers and a full wave;
    # every key three times with at most two values kept
    keys = o.gen_unique_keys(kb, 148 * 4 * 256 + 1, 80)
    for n in (1, 31, 32, 33, 63, 64, 65, 96, 97, len(keys)):
        t = wc.MultiValueHashTable(4 * n, key_bytes=kb, value_bytes=vb, max_values_per_key=2,
                                   cg_size=cg)
        st = empty_dev(n, 4)
        for round_, expect in enumerate((0, 1 << 4, (1 << 4) | (1 << 11))):
            vals = (np.arange(n) + 1 + round_ * n).astype(DT[vb])
            t.insert(dev(keys[:n]), dev(vals), status_out=st)
            assert (host(st) == expect).all()
        assert t.num_keys() == n and t.size() == 2 * n
        num, b, e, v, _ = retrieve(t, keys[:n], 2 * n, vb)
        assert num == 2 * n
        got = v.view(DT[vb]).reshape(n, 2)
        assert np.array_equal(got[:, 0], np.arange(n) + 1)
        assert np.array_equal(got[:, 1], np.arange(n) + 1 + n)


@pytest.mark.parametrize("kb,vb,cg", [(4, 4, 8), (8, 8, 8), (4, 8, 4), (8, 4, 16)])
def test_bucket_list_insert_sizes(kb, vb, cg):
    # one key per resident lane and one more (the line between the two
    # kernels), full and ragged tiles; equal keys in one batch; a limit
    # of values per key; a pool that runs out; keys without a slot
    wave = 148 * 4 * 256
    keys = o.gen_unique_keys(kb, wave + 1, 81)
    for n, per in ((wave, 1), (wave + 1, 1), (wave // 5 + 7, 7), (2 * kb + 3, wave // 8)):
        t = wc.BucketListHashTable(2 * n, 4 * n * per, key_bytes=kb, value_bytes=vb, cg_size=cg)
        at = np.random.default_rng(9).permutation(np.repeat(np.arange(n), per))
        vals = (np.arange(n * per) + 1).astype(DT[vb])
        st = empty_dev(n * per, 4)
        t.insert(dev(keys[at]), dev(vals), status_out=st)
        assert t.num_keys() == n and t.num_values() == n * per
        assert np.count_nonzero(host(st) == 0) == n  # one claim per key
        assert np.count_nonzero(host(st) == 1 << 4) == n * (per - 1)
        num, b, e, v, _ = retrieve(t, keys[:n], n * per, vb)
        assert num == n * per
        owner = np.repeat(np.arange(n), e - b)
        order = np.argsort(v.view(DT[vb]), kind="stable")
        assert np.array_equal(v.view(DT[vb])[order], vals)
        assert np.array_equal(owner[order], at)
    n = wave + 1
    t = wc.BucketListHashTable(2 * n, 4 * n, key_bytes=kb, value_bytes=vb, cg_size=cg,
                               max_values_per_key=1)
    st = empty_dev(n, 4)
    for expect in (0, (1 << 4) | (1 << 11)):
        t.insert(dev(keys), dev((np.arange(n) + 1).astype(DT[vb])), status_out=st)
        assert (host(st) == expect).all()
    small = wc.BucketListHashTable(2 * n, n // 2, key_bytes=kb, value_bytes=vb, cg_size=cg)
    small.insert(dev(keys), dev((np.arange(n) + 1).astype(DT[vb])), status_out=st)
    got = host(st)
    assert set(np.unique(got)) == {0, 1 << 7}
    assert np.count_nonzero(got == 0) == small.num_values() <= n // 2
    few = wc.BucketListHashTable(1000, 4 * n, key_bytes=kb, value_bytes=vb, cg_size=cg)
    many = o.gen_unique_keys(kb, few.key_capacity + n, 82)
    st = empty_dev(len(many), 4)
    few.insert(dev(many), dev((np.arange(len(many)) + 1).astype(DT[vb])), status_out=st,
               probing_length=cg)
    got = host(st)
    assert set(np.unique(got)) <= {0, 1 << 1, 1 << 7}
    assert np.count_nonzero(got & 2) == len(many) - few.num_keys()


@pytest.mark.parametrize("kb,vb,cg", [(4, 4, 8), (8, 8, 8), (4, 8, 16), (8, 4, 4)])
@pytest.mark.parametrize("bucket", [1, 2, 3, 4])
def test_multi_bucket_insert_sizes(kb, vb, cg, bucket):
    # input counts around a warp, its queue of 64 and a full wave; equal keys
    # in one batch; a limit of values per key; the empty value; full windows
    keys = o.gen_unique_keys(kb, 148 * 4 * 256 + 1, 83)
    for n, per in ((1, 1), (31, 1), (33, 2), (64, 3), (97, 2), (len(keys), 1), (30011, 5)):
        t = wc.MultiBucketHashTable(2 * n * per, key_bytes=kb, value_bytes=vb, bucket_size=bucket,
                                    cg_size=cg)
        at = np.random.default_rng(9).permutation(np.repeat(np.arange(n), per))
        vals = (np.arange(n * per) + 1).astype(DT[vb])
        st = empty_dev(n * per, 4)
        t.insert(dev(keys[at]), dev(vals), status_out=st)
        assert t.num_keys() == n and t.size() == n * per
        assert np.count_nonzero(host(st) == 0) == n  # one first value per key
        assert np.count_nonzero(host(st) == 1 << 4) == n * (per - 1)
        num, b, e, v, _ = retrieve(t, keys[:n], n * per, vb)
        assert num == n * per
        owner = np.repeat(np.arange(n), e - b)
        order = np.argsort(v.view(DT[vb]), kind="stable")
        assert np.array_equal(v.view(DT[vb])[order], vals)
        assert np.array_equal(owner[order], at)
    n = 5003
    t = wc.MultiBucketHashTable(4 * n, key_bytes=kb, value_bytes=vb, bucket_size=bucket,
                                cg_size=cg, max_values_per_key=2)
    st = empty_dev(n, 4)
    for expect in (0, 1 << 4, (1 << 4) | (1 << 11)):
        t.insert(dev(keys[:n]), dev((np.arange(n) + 1).astype(DT[vb])), status_out=st)
        assert (host(st) == expect).all()
    t.insert(dev(keys[:n]), dev(np.zeros(n, dtype=DT[vb])), status_out=st)
    assert (host(st) == 1 << 12).all()  # invalid_value
    few = wc.MultiBucketHashTable(1000, key_bytes=kb, value_bytes=vb, bucket_size=bucket, cg_size=cg)
    many = o.gen_unique_keys(kb, few.capacity + n, 84)
    st = empty_dev(len(many), 4)
    few.insert(dev(many), dev((np.arange(len(many)) + 1).astype(DT[vb])), status_out=st,
               probing_length=cg)
    got = host(st)
    assert set(np.unique(got)) == {0, 1 << 1}
    assert np.count_nonzero(got == 0) == few.num_keys() == few.num_occupied()
