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
