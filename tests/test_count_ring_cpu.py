"""The ring of (value, sequence number) pairs that kernels fill in: what the host makes of a pair that was used again, with the
kernels' two stores done by the test."""
import ctypes as C

import torch

from starrygl import _C


def ring():
    r = _C.CountRing()
    r._buf = torch.zeros(2 * r.SLOTS, dtype=torch.int64)
    r._base = r._buf.data_ptr()
    r._words = (C.c_int64 * (2 * r.SLOTS)).from_address(r._base)
    return r


def arrive(r, taken, value):
    r._words[taken[1]] = value
    r._words[taken[1] + 1] = taken[2]


def test_value_of_a_pair_that_is_being_overwritten_is_not_taken_for_the_old_one():
    r = ring()
    first = r.take()
    arrive(r, first, 5)
    assert r.value(first, None) == 5
    for _ in range(r.SLOTS - 1):
        t = r.take()
        arrive(r, t, 7)
        assert r.value(t, None) == 7
    again = r.take()
    assert again[1] == first[1]
    r._words[again[1]] = 9                   # the value's store is there, the sequence number's not yet
    assert r.value(first, None) is None
    arrive(r, again, 9)
    assert r.value(again, None) == 9 and r.value(first, None) is None


def test_a_pair_whose_count_is_still_to_come_is_not_given_out_again():
    r = ring()
    late = r.take()
    for _ in range(r.SLOTS - 1):
        arrive(r, r.take(), 1)
    assert r.take() is None
    arrive(r, late, 3)
    assert r.value(late, None) == 3
    others = [r.take() for _ in range(r.SLOTS)]
    assert all(others) and others[-1][1] == late[1]


def test_pairs_of_failed_calls_are_given_out_again():
    r = ring()
    for _ in range(2 * r.SLOTS):
        t = r.take()
        assert t is not None
        r.give_back(t)
