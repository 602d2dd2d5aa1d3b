"""Lists at and above the mini-batch sort's capacity (1,212,416 entries), where radix passes and the delivery kernel take over, for
every operation on lists; the forms of a T-CSR build of that size; route plans on both sides of 32 ranks."""
import numpy as np
import pytest
import torch

from oracle import oracle_np as O
from gpu_util import cu, npy

pytestmark = pytest.mark.gpu

LIMIT = 148 * 8192
SIZES = [LIMIT, LIMIT + 1, LIMIT + 70001]


@pytest.mark.parametrize("n", SIZES)
def test_pairs_and_relabel(n):
    from starrygl import ops
    rng = np.random.default_rng(n)
    ids, ts = rng.integers(0, 50000, n).astype(np.int64), rng.integers(-20, 20, n).astype(np.int64)
    cut = n // 5
    st = ops.StatusWord(torch.device("cuda"))
    out_id, out_ts, inv_a, inv_b, d_n = ops.unique_pairs(cu(ids[:cut]), cu(ts[:cut]), cu(ids[cut:]), cu(ts[cut:]), id_bits=16, ts_bits=6,
                                                         ts_base=-20, status=st)[:5]
    uniq, inv = np.unique((ids << 6) | (ts + 20), return_inverse=True)
    assert int(d_n) == len(uniq)
    assert np.array_equal(npy(out_id[:len(uniq)]), uniq >> 6) and np.array_equal(npy(out_ts[:len(uniq)]), (uniq & 63) - 20)
    assert np.array_equal(npy(inv_b[:n - cut]), inv[cut:])
    rl = ops.NodeRelabeler(60000, torch.device("cuda"))
    known = {}
    for lst in (ids, rng.integers(0, 60000, n).astype(np.int64)):
        loc, new, d_new = rl.insert(cu(lst), status=st)
        fresh = np.setdiff1d(np.unique(lst), np.fromiter(known, np.int64, len(known)))
        base = len(known)
        known.update((int(g), base + i) for i, g in enumerate(fresh))
        table = np.full(60000, -1, np.int64)
        table[np.fromiter(known.keys(), np.int64)] = np.fromiter(known.values(), np.int64)
        assert int(d_new) == len(fresh) and np.array_equal(npy(new[:len(fresh)]), fresh) and np.array_equal(npy(loc), table[lst])
    st.check("lists")


@pytest.mark.parametrize("n", SIZES)
def test_csc_and_newest_entry(n):
    from starrygl import ops
    rng = np.random.default_rng(n)
    rows = 30000
    dst, ts = rng.integers(0, rows, n).astype(np.int64), rng.integers(0, 1000, n).astype(np.int64)
    src, eid, dt = rng.integers(0, 9, n).astype(np.int64), np.arange(n, dtype=np.int64), rng.standard_normal(n).astype(np.float32)
    got = ops.build_csc(cu(src), cu(dst), None, cu(ts), cu(dt), cu(eid), rows, dst_bits=15, ts_bits=10, ts_base=0)
    want = O.build_csc(src, dst, ts, dt, eid, rows)
    for a, b in zip(got, want):
        assert np.array_equal(npy(a), b)
    fts = rng.integers(-50, 50, n).astype(np.float32)
    index, _, out_ts, pos, d_u = ops.mail_reduce(cu(dst), None, cu(fts), rows, want_pos=True)
    order = np.lexsort((np.arange(n), -fts, dst))
    first = order[np.unique(dst[order], return_index=True)[1]]
    u = int(d_u)
    assert u == len(first) and np.array_equal(npy(pos[:u]), first) and np.array_equal(npy(index[:u]), dst[first])
    assert np.array_equal(npy(out_ts[:u]), fts[first])


@pytest.mark.parametrize("m", [LIMIT, LIMIT + 1, LIMIT + 50000])
@pytest.mark.parametrize("ordered", [False, True])
@pytest.mark.parametrize("form", ["ids", "no ids", "wide ids", "positions"])
def test_tcsr_forms(m, ordered, form):
    from starrygl import ops
    rng = np.random.default_rng(m)
    n = 70001
    key, nbr = rng.integers(0, n, m).astype(np.int64), rng.integers(0, n, m).astype(np.int64)
    ts = rng.integers(-10 ** 6, 10 ** 6, m).astype(np.int64)
    if ordered:
        ts.sort()
    eid = None if form == "no ids" else rng.integers(0, 2 ** 31, m).astype(np.int64)
    if form == "wide ids":
        eid[m // 2] = 2 ** 40
    g = ops.tcsr_build(cu(key), cu(nbr), cu(ts), None if eid is None else cu(eid), n, want_perm=form == "positions")
    indptr, o_nbr, o_ts, o_eid, order = O.tcsr_build(key, nbr, ts, np.arange(m, dtype=np.int64) if eid is None else eid, n)
    for a, b in ((g.indptr, indptr), (g.nbr, o_nbr), (g.ts, o_ts), (g.eid, o_eid)):
        assert np.array_equal(npy(a), b)
    if form == "positions":
        assert np.array_equal(npy(g.perm), order)


def test_tcsr_two_rounds_of_passes():
    """Node and timestamp bits above 64, beyond the mini-batch limit."""
    from starrygl import ops
    rng = np.random.default_rng(2)
    n, m = 1 << 20, LIMIT + 3
    key, ts = rng.integers(0, n, m).astype(np.int64), rng.integers(-2 ** 62, 2 ** 62, m, dtype=np.int64)
    ts[:1000] = ts[1000:2000]
    g = ops.tcsr_build(cu(key), cu(key), cu(ts), None, n)
    indptr, o_nbr, o_ts, o_eid, _ = O.tcsr_build(key, key, ts, np.arange(m, dtype=np.int64), n)
    for a, b in ((g.indptr, indptr), (g.nbr, o_nbr), (g.ts, o_ts), (g.eid, o_eid)):
        assert np.array_equal(npy(a), b)


@pytest.mark.parametrize("ranks", [2, 31, 32, 33, 60])
@pytest.mark.parametrize("n", [1, 255, 257, 9000])
def test_route_plan_ranks(ranks, n):
    from starrygl.cache.cache_route import compute_layer_route
    from starrygl.cache.replica_table import CSRReplicaTable
    rng = np.random.default_rng(ranks + n)
    nodes = 3000
    parts = rng.integers(0, ranks, nodes).astype(np.int64)
    book = [rng.choice(nodes, int(rng.integers(0, 400)), replace=False) for _ in range(ranks)]
    indptr, rep_ranks, rep_locs = O.build_replica_table(nodes, book)
    ids = np.sort(rng.integers(0, nodes, n)).astype(np.int64)       # a layer list: by node, then time
    times = np.arange(n, dtype=np.int64)
    plan = compute_layer_route(cu(ids), cu(parts), 1, CSRReplicaTable(cu(indptr), cu(rep_ranks), cu(rep_locs)), ranks)
    ref = O.compute_layer_route(ids, times, parts, 1, indptr, rep_ranks, rep_locs, ranks)
    if ref is None:
        assert plan is None
        return
    for a, b in zip((plan.send_ranks, plan.send_sizes, plan.send_indices, plan.send_remote_indices), ref):
        assert np.array_equal(npy(a), b)


@pytest.fixture
def no_patience():
    """Look-backs of this thread's calls give up at once."""
    from starrygl import _C
    before = _C.lib().sgl_look_back_limit(0)
    yield
    _C.lib().sgl_look_back_limit(before)


def _big_build(form, m=8_000_000):
    from starrygl import ops
    gen = torch.Generator(device="cuda").manual_seed(3)
    wide = 2 ** 62 if form == "two rounds" else 100_000
    key, nbr = (torch.randint(0, 50_000, (m,), device="cuda", generator=gen) for _ in range(2))
    ts = torch.randint(0, wide, (m,), device="cuda", generator=gen)
    return key, ops.tcsr_build(key, nbr, ts, None, 50_000, want_perm=form != "pairs")


@pytest.mark.parametrize("form", ["pairs", "positions", "two rounds"])
def test_build_whose_sort_gives_up_raises(form, no_patience):
    from starrygl import _C
    with pytest.raises(_C.SglError, match="time limit"):
        _big_build(form)
    _C.lib().sgl_look_back_limit(2_000_000_000)
    key, g = _big_build(form)
    assert torch.equal(g.indptr[1:] - g.indptr[:-1], torch.bincount(key, minlength=50_000))


def test_sort_and_lists_that_give_up_say_so(no_patience):
    from starrygl import _C, ops
    n = 8_000_000
    keys = torch.randint(0, 2 ** 40, (n,), device="cuda")
    with pytest.raises(_C.SglError, match="time limit"):
        ops.radix_sort_pairs(keys, torch.arange(n, dtype=torch.int32, device="cuda"), 40)
    st = ops.StatusWord(keys.device)
    ops.unique_pairs(keys, torch.zeros_like(keys), id_bits=40, ts_bits=0, ts_base=0, status=st)
    with pytest.raises(_C.SglError, match="device status"):
        st.check("lists")
