"""Results of the step-by-step path: sizes are read once for all hops; copies and files of results and hops stand on their own; nobody holds
anybody else's arrays."""
import copy
import gc
import io
import pickle
import weakref

import pytest
import torch

from starrygl import _C, ops
from starrygl.lib.libstarrygl_comm import TemporalNeighbor, TemporalResult, TemporalRoot

SIZES = [7, 5, 2]


def hop(n, queries, cap=20):
    a = torch.arange(cap)
    return ops.Hop(a.clone(), a.clone(), a.clone(), a.float(), a.clone(), torch.tensor([0] * queries + [n]), cap, a.clone())


def result(status=True):
    r = torch.arange(3)
    out = TemporalResult(TemporalRoot(r, torch.arange(4), r))
    if status:
        out._status = ops.StatusWord("cpu")
    for l, n in enumerate(SIZES):
        out.neighbors_list.append(TemporalNeighbor(hop(n, 3 if l == 0 else 20), out, 3 if l == 0 else None))
    return out


def check(nb, l):
    assert nb.neighbor_num == SIZES[l] and nb.neighbors.numel() == nb.neighbors_ts.numel() == SIZES[l]
    assert nb.root_start_ptr.numel() == (3 if l == 0 else SIZES[l - 1]) + 1


COPIES = {"pickle": lambda x: pickle.loads(pickle.dumps(x)), "deepcopy": copy.deepcopy, "copy": copy.copy}


def through_a_file(x):
    f = io.BytesIO()
    torch.save(x, f)
    f.seek(0)
    return torch.load(f, weights_only=False)


COPIES["file"] = through_a_file


@pytest.mark.parametrize("how", COPIES)
@pytest.mark.parametrize("known", [False, True])
def test_copies(how, known):
    out = result()
    if known:
        out.materialize()
    for l, nb in enumerate(COPIES[how](out).neighbors_list):
        check(nb, l)
    for l in range(3):
        check(COPIES[how](result().neighbors_list[l]), l)
    for l, nb in enumerate(out.neighbors_list):
        check(nb, l)


@pytest.mark.parametrize("order", [(0, 1, 2), (2, 1, 0), (1, 0, 2)])
def test_hops_without_their_result(order):
    hops = result().neighbors_list
    for l in order:
        check(hops[l], l)
    assert all(hops[l].hop.nbr.numel() == 20 for l in order)


@pytest.mark.parametrize("cut", [False, True])
def test_a_hop_keeps_no_other(cut):
    gc.collect()
    gc.disable()
    try:
        out = result()
        last, first = out.neighbors_list[-1], weakref.ref(out.neighbors_list[0])
        arrays = weakref.ref(out.neighbors_list[1].hop.nbr)
        if cut:
            check(last, 2)
        del out
        assert first() is None and arrays() is None
        check(last, 2)
    finally:
        gc.enable()


def test_error_bits_ride_along():
    out = result()
    out._status.t.fill_(4)
    with pytest.raises(_C.SglError, match="row index out of range"):
        out.neighbors_list[1].neighbor_num
    for l, nb in enumerate(out.neighbors_list):       # (reported once)
        check(nb, l)


@pytest.mark.parametrize("first", ["map", "hops"])
def test_remap_pieces_come_in_the_same_copy(monkeypatch, first):
    out = result()
    out._remap_pieces = [(torch.arange(a, a + 10), out._sizes.add(torch.tensor([n]))) for a, n in ((10, 4), (30, 0), (50, 2))]
    copies = []
    real = torch.Tensor.tolist
    monkeypatch.setattr(torch.Tensor, "tolist", lambda t: copies.append(1) or real(t))
    if first == "map":
        assert torch.equal(out.nodes_remapper_id, torch.tensor([10, 11, 12, 13, 50, 51]))
    for l, nb in enumerate(out.neighbors_list):
        check(nb, l)
    assert torch.equal(out.nodes_remapper_id, torch.tensor([10, 11, 12, 13, 50, 51]))
    assert len(copies) == 1 and out._remap_pieces == []
