"""Counting inserts without statuses on each kernel that serves them: one count
cache per SM (default), groups of lanes per window, fingerprints first.  The
parity suites' small tables all take the first, so the tests of the count
caches are collected again here with wc_lane_ops bit 1 clear."""
import numpy as np
import pytest

import warpcore_b200 as wc
from oracle import oracle as o
from tests.test_counting_cache_gpu import test_counts  # noqa: F401  (re-collected below)
from tests.test_tables_gpu import test_counting_cache_and_direct_claims_agree  # noqa: F401
from tests.wc_helpers import dev, empty_dev, host

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, params=["cache per SM", "groups", "fingerprints"])
def path(request):
    prev = wc.set_lane_ops(0xF if request.param == "cache per SM" else 0xD)
    policy = wc.set_fingerprint_policy("always" if request.param == "fingerprints" else "auto")
    yield request.param
    wc.set_fingerprint_policy(policy)
    wc.set_lane_ops(prev)


def test_switch():
    # the counting bit is kept and on by default (the fixture has set it)
    now = wc.set_lane_ops(0xF)
    assert now in (0xF, 0xD)
    assert wc.set_lane_ops(2) == 0xF
    assert wc.set_lane_ops(now) == 2


@pytest.mark.parametrize("kb", [4, 8])
def test_statuses_of_full_tables(kb, path):
    # more distinct keys than slots, four windows each: a key is counted whole
    # or not at all, and the table's status says that some were not
    t = wc.CountingHashTable(1000, key_bytes=kb, value_bytes=4, cg_size=8)
    n = t.capacity + 50_000
    keys = o.gen_unique_keys(kb, n, 97)
    t.insert(dev(np.repeat(keys, 3)), probing_length=32)
    assert int(t.pop_status()) == o.ST_DUPLICATE_KEY | o.ST_PROBING_LENGTH_EXCEEDED
    out = empty_dev(n, 4)
    t.retrieve(dev(keys), out)
    got = host(out)
    assert set(np.unique(got)) == {0, 3}
    assert np.count_nonzero(got) == t.size() == t.size_scan()
    assert t.capacity * 3 // 4 < t.size() < t.capacity
