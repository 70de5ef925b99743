"""Lookups of several values per key at window widths chosen at run time, query
counts around the tiles of 1024 keys and the waves of both halves."""
import numpy as np
import pytest
import torch

import warpcore_b200 as wc
from oracle import oracle as o
from tests.wc_helpers import dev, empty_dev, host

pytestmark = pytest.mark.gpu

DT = {4: np.uint32, 8: np.uint64}


@pytest.mark.parametrize("kind", ["mv", "mb", "bl"])
@pytest.mark.parametrize("kb,vb,cg", [(4, 4, 4), (4, 8, 16), (4, 4, 32), (8, 4, 2), (8, 8, 32)])
def test_counts_and_values(kind, kb, vb, cg):
    nkeys, per = 3000, 3
    both = o.gen_unique_keys(kb, 2 * nkeys, 101)
    if kind == "mv":
        t = wc.MultiValueHashTable(2 * nkeys * per, key_bytes=kb, value_bytes=vb, cg_size=cg)
    elif kind == "mb":
        t = wc.MultiBucketHashTable(2 * nkeys * per, key_bytes=kb, value_bytes=vb, cg_size=cg,
                                    bucket_size=2)
    else:
        t = wc.BucketListHashTable(2 * nkeys, 4 * nkeys * per, key_bytes=kb, value_bytes=vb,
                                   cg_size=cg)
    rng = np.random.default_rng(13)
    values = rng.integers(1, 2**31, size=(nkeys, per)).astype(DT[vb])
    for j in range(per):
        t.insert(dev(both[:nkeys]), dev(np.ascontiguousarray(values[:, j])))
    for n in (1, 1023, 1024, 1025, 2049, 148 * 5 * 1024 + 1, 148 * 6 * 1024 + 1025):
        at = rng.integers(0, 2 * nkeys, size=n)
        at[::101] = -1  # the reserved key among the queries
        q = both[at]
        q[::101] = t.info().empty_key
        hit = (at >= 0) & (at < nkeys)
        cnt = np.where(hit, per, 0)
        st = empty_dev(n, 4)
        counts = torch.full((n,), -7, dtype=torch.int64, device="cuda")
        assert t.num_values(dev(q), counts, status_out=st) == cnt.sum()
        assert np.array_equal(host(counts).astype(np.int64), cnt)
        want = np.where(hit, 0, np.where(at < 0, o.ST_INVALID_KEY, o.ST_KEY_NOT_FOUND))
        assert np.array_equal(host(st), want)
        assert t.num_values(dev(q)) == cnt.sum()
        begin, end = (torch.full((n,), -7, dtype=torch.int64, device="cuda") for _ in range(2))
        out = empty_dev(max(int(cnt.sum()), 1), vb)
        assert t.retrieve(dev(q), begin, end, out, status_out=st) == cnt.sum()
        assert np.array_equal(host(end).astype(np.int64), np.cumsum(cnt))
        assert np.array_equal(host(begin).astype(np.int64), np.cumsum(cnt) - cnt)
        assert np.array_equal(host(st), want)
        got = host(out)[:cnt.sum()].reshape(-1, per)
        assert np.array_equal(np.sort(got, axis=1), np.sort(values[at[hit]], axis=1))
