"""T-CSR builds by radix passes (above 1,212,416 edges): ids beyond 32 bits anywhere in the input, among the first and last 303,104 edges that
the scan looks at or between them; skewed and ordered keys, for which a warp's digits are counted together."""
import numpy as np
import pytest
import torch

from starrygl import ops

pytestmark = pytest.mark.gpu
M = 1_212_417


def check(key, nbr, ts, eid, nodes):
    cu = lambda a: torch.from_numpy(a).cuda()
    g = ops.tcsr_build(cu(key), cu(nbr), cu(ts), None if eid is None else cu(eid), nodes)
    order = np.lexsort((ts, key))
    assert np.array_equal(g.nbr.cpu().numpy(), nbr[order])
    assert np.array_equal(g.ts.cpu().numpy(), ts[order])
    assert np.array_equal(g.eid.cpu().numpy(), order if eid is None else eid[order])
    assert np.array_equal(g.indptr.cpu().numpy(), np.searchsorted(key[order], np.arange(nodes + 1)))


@pytest.mark.parametrize("which", ["nbr", "eid"])
@pytest.mark.parametrize("place", [0, 303_103, 303_104, 900_001, M - 1])
def test_wide_ids(which, place):
    rng = np.random.default_rng(place)
    key, nbr, ts, eid = rng.integers(0, 70_000, M), rng.integers(0, 1 << 32, M), rng.integers(0, 1 << 24, M), np.arange(M)
    (nbr if which == "nbr" else eid)[place] = 1 << 32 if place % 2 else -1
    check(key, nbr, ts, eid, 70_000)


@pytest.mark.parametrize("kind", ["ordered", "one node", "hub", "blocks"])
def test_counts_of_alike_digits(kind):
    rng = np.random.default_rng(7)
    key, ts = rng.integers(0, 70_000, M + 33), rng.integers(0, 1 << 24, M + 33)
    if kind == "ordered":
        ts.sort()
    elif kind == "one node":
        key[:] = 69_999
    elif kind == "hub":
        key[rng.random(key.size) < 0.6] = 41
    else:                                     # warps whose first keys are alike and others that are not
        key[(np.arange(key.size) // 512) % 3 == 0] = 5
    check(key, rng.integers(0, 70_000, key.size), ts, None, 70_000)
