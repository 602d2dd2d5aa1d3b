"""CSC of the later hops along the layer list's order: rows of one and of several targets, rows at and above the number of
targets from which the sort takes over, fan-outs with and without the edge-to-item map, recent and uniform."""
import numpy as np
import pytest
import torch

from oracle import oracle_np as O
from gpu_util import cu, npy, build_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("queries", [1, 31, 32, 33, 400])
@pytest.mark.parametrize("fanouts", [[3, 4], [3, 40], [2, 3, 5]])
@pytest.mark.parametrize("policy", ["recent", "uniform"])
def test_rows_of_many_targets(queries, fanouts, policy):
    from starrygl.graph.batch import build_batch
    rng = np.random.default_rng(queries)
    n, m = 200, 6000
    # node 0 has three events, so every later query of it samples them all: one pair per event, `queries` targets each
    src = np.concatenate([rng.integers(2, n, m), [1, 5, 1]]).astype(np.int64)
    dst = np.concatenate([rng.integers(1, n, m), [0, 0, 0]]).astype(np.int64)
    ts = np.concatenate([np.sort(rng.integers(0, 500, m)), [400, 420, 430]]).astype(np.int64)
    z = {"n": n, "dst": dst, "src": src, "ts": ts, "eid": np.arange(m + 3, dtype=np.int64)}
    g = build_graph(z)
    indptr, nbr, tss, eid, _ = O.tcsr_build(dst, src, ts, z["eid"], n)
    roots = np.concatenate([np.zeros(queries, np.int64), rng.integers(1, n, 250)])
    rts = np.concatenate([600 + np.arange(queries), rng.integers(100, 500, 250)]).astype(np.int64)
    pol = O.RECENT if policy == "recent" else O.UNIFORM
    ref = O.build_batch(indptr, nbr, tss, eid, roots, rts, fanouts, pol, seed=3)
    out = build_batch(g, cu(roots), cu(rts), fanouts, policy, seed=3, ts_range=(0, 1100))
    assert len(out) == len(ref)
    for i, (d, r) in enumerate(zip(out, ref)):
        for k in r:
            a = npy(d[k])
            assert a.dtype == r[k].dtype and np.array_equal(a, r[k]), (i, k)


@pytest.mark.parametrize("copies, fanouts", [(50, [20, 20]), (50, [20, 21]), (50, [20, 21, 2])])
def test_narrow_columns(copies, fanouts):
    """Both sides of the capacity from which the merge scatters 32-bit positions (8 Mi edges), and a hop behind it."""
    from starrygl.graph.batch import build_batch
    rng = np.random.default_rng(1)
    n, m = 300, 2500
    src, dst = rng.integers(0, n, m).astype(np.int64), rng.integers(0, n, m).astype(np.int64)
    ts = np.sort(rng.integers(0, 900, m)).astype(np.int64)
    z = {"n": n, "dst": dst, "src": src, "ts": ts, "eid": np.arange(m, dtype=np.int64)}
    g = build_graph(z)
    indptr, nbr, tss, eid, _ = O.tcsr_build(dst, src, ts, z["eid"], n)
    roots = np.tile(rng.integers(0, n, 400), copies).astype(np.int64)
    rts = np.tile(rng.integers(100, 1000, 400), copies).astype(np.int64)
    ref = O.build_batch(indptr, nbr, tss, eid, roots, rts, fanouts, O.UNIFORM, seed=4)
    out = build_batch(g, cu(roots), cu(rts), fanouts, "uniform", seed=4, ts_range=(0, 1000))
    assert len(out) == len(ref)
    for i, (d, r) in enumerate(zip(out, ref)):
        for k in r:
            assert np.array_equal(npy(d[k]), r[k]), (i, k)


def test_sort_that_is_needed_after_all_of_millions_of_edges():
    """Rows of more targets than the rows kernel takes, in a hop of more edges than the sort's passes have CTAs for at a time (2,121,728):
    its CTAs take a second tile, and what the first one left in shared memory is gone."""
    from starrygl import ops
    from starrygl.graph.batch import build_batch_async
    gen = torch.Generator(device="cuda").manual_seed(2)
    n, m, roots, fanouts = 1000, 300_000, 4000, [30, 50]
    src, dst = (torch.randint(0, n, (m,), device="cuda", generator=gen) for _ in range(2))
    g = ops.tcsr_build(src, dst, torch.randint(0, 4, (m,), device="cuda", generator=gen), None, n)
    db = build_batch_async(g, torch.arange(roots, device="cuda") % n, 4 + torch.arange(roots, device="cuda"), fanouts, "uniform",
                           ts_range=(0, 4 + roots))
    out = db.finish()
    first, hop = db.layers[1], db.layers[2]["hop"]
    k, targets = int(db.counts[3]), int(db.counts[1])
    assert k > 2 * 2_121_728
    per_target = hop.offsets[1:targets + 1] - hop.offsets[:targets]
    assert int(torch.bincount(first["inv"][:targets][per_target == fanouts[1]]).max()) > 33
    row, ts = first["inv"][hop.dst[:k]], hop.ts[:k]
    order = torch.sort(row * 8 + ts, stable=True).indices
    rows = out[1]["gids"].numel()
    assert torch.equal(out[2]["indptr"], torch.cat([row.new_zeros(1), torch.bincount(row, minlength=rows).cumsum(0)]))
    for name, raw in (("indices", db.layers[2]["inv"]), ("eid", hop.eid), ("edge_ts", hop.ts), ("edge_dt", hop.dt)):
        assert torch.equal(out[2][name], raw[:k][order]), name


def test_neighbours_outside_the_graph_are_an_error():
    """A list entry of replaced ids has targets with different edges: rows of the CSC stay partly unwritten, the call raises."""
    from starrygl import _C, ops
    from starrygl.graph.batch import build_batch
    n, per = 256, 40
    rng = np.random.default_rng(0)
    key = np.repeat(np.arange(n), per)
    ts = np.tile(np.arange(per) // 4, n)                       # four edges of every node at each time
    good = rng.integers(0, n, n * per)
    bad = np.where(np.arange(n * per) % 2 == 0, 0, 2 ** 30)   # node 0 and an id that becomes node 0, at the same times
    q, qt = torch.arange(n).cuda().repeat(4), torch.full((4 * n,), per).cuda()
    for nbr in (bad, good):
        g = ops.tcsr_build(cu(key), cu(nbr.astype(np.int64)), cu(ts), None, n)
        junk = [torch.full((1 << k,), 2 ** 61, device="cuda") for k in range(15, 25) for _ in range(4)]   # what memory holds before
        del junk
        if nbr is bad:
            with pytest.raises(_C.SglError, match="node id out of range, row index out of range"):
                build_batch(g, q, qt, [10, 10], "recent")
        else:
            assert len(build_batch(g, q, qt, [10, 10], "recent")) == 3
