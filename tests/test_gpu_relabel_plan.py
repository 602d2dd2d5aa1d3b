"""Node relabel at the edges of its bitmap form (list length, number of nodes, ids out of range, lists that continue each other), route
plans whose nodes have more copies than a shared scan holds, and batches that are laid out while their last list is merged."""
import numpy as np
import pytest
import torch

from oracle import oracle_np as O
from gpu_util import cu, npy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_nodes", [1, 32, 33, 2048, 70001, 2 ** 19, 2 ** 19 + 1])
@pytest.mark.parametrize("n", [2048, 2049, 30000])
def test_relabel_of_lists_that_continue_each_other(num_nodes, n):
    from starrygl import ops
    rng = np.random.default_rng(num_nodes + n)
    rl = ops.NodeRelabeler(num_nodes, torch.device("cuda"))
    st = ops.StatusWord(torch.device("cuda"))
    for epoch in range(2):
        table, base = np.full(num_nodes, -1, np.int64), 0
        for part in range(3):
            ids = rng.integers(0, max(num_nodes * (part + 1) // 3, 1), n).astype(np.int64)
            used = n if part != 1 else n // 3                  # (a count on the device, below the capacity)
            d_n = None if part != 1 else torch.tensor([used], device="cuda")
            local, new, d_new = rl.insert(cu(ids), d_n=d_n, status=st)
            fresh = np.unique(ids[:used])
            fresh = fresh[table[fresh] < 0]
            table[fresh] = base + np.arange(len(fresh))
            base += len(fresh)
            assert int(d_new) == len(fresh) and np.array_equal(npy(new[:len(fresh)]), fresh)
            assert np.array_equal(npy(local[:used]), table[ids[:used]]) and int(rl.next_local) == base
        rl.reset()
    st.check("relabel")


@pytest.mark.parametrize("num_nodes", [32, 50000])
@pytest.mark.parametrize("share", [0.5, 0.99, 1.0])
def test_relabel_of_lists_with_hubs(num_nodes, share):
    """Nodes that a large part of the list is copies of: all lanes of a warp, and all warps, mark the same word."""
    from starrygl import ops
    rng = np.random.default_rng(num_nodes)
    n = 1_300_000
    rl, st = ops.NodeRelabeler(num_nodes, torch.device("cuda")), ops.StatusWord(torch.device("cuda"))
    table, base = np.full(num_nodes, -1, np.int64), 0
    for hubs in ([7], [0, 31, num_nodes - 1]):
        ids = np.where(rng.random(n) < share, rng.choice(hubs, n), rng.integers(0, num_nodes, n)).astype(np.int64)
        local, new, d_new = rl.insert(cu(ids), status=st)
        fresh = np.unique(ids)
        fresh = fresh[table[fresh] < 0]
        table[fresh] = base + np.arange(len(fresh))
        base += len(fresh)
        assert int(d_new) == len(fresh) and np.array_equal(npy(new[:len(fresh)]), fresh) and np.array_equal(npy(local), table[ids])
    st.check("relabel")


def test_relabel_flags_ids_out_of_range():
    from starrygl import ops
    n, num_nodes = 5000, 1000
    ids = np.arange(n, dtype=np.int64) % num_nodes
    ids[[3, 4000]] = [-1, num_nodes]
    rl, st = ops.NodeRelabeler(num_nodes, torch.device("cuda")), ops.StatusWord(torch.device("cuda"))
    local, _, d_new = rl.insert(cu(ids), status=st)
    with pytest.raises(Exception, match="status"):
        st.check("relabel")
    want = ids.copy()
    want[[3, 4000]] = -1
    assert int(d_new) == num_nodes and np.array_equal(npy(local), want)


@pytest.mark.parametrize("num_parts", [2, 4, 5, 32])
@pytest.mark.parametrize("copies", [3, 255, 256, 700])
def test_route_plan_of_nodes_with_many_copies(num_parts, copies):
    from starrygl.cache.cache_route import compute_layer_route
    from starrygl.cache.replica_table import CSRReplicaTable
    rng = np.random.default_rng(copies * num_parts)
    nodes = 900
    parts = rng.integers(0, num_parts, nodes).astype(np.int64)
    counts = np.where(rng.random(nodes) < 0.02, copies, rng.integers(0, 4, nodes))
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    ranks = rng.integers(0, num_parts, indptr[-1]).astype(np.int64)
    one = rng.random(nodes) < 0.5                              # (all copies on one rank)
    for v in np.nonzero(one)[0]:
        ranks[indptr[v]:indptr[v + 1]] = rng.integers(0, num_parts)
    locs = np.arange(indptr[-1], dtype=np.int64)
    ids = np.sort(rng.integers(0, nodes, 5000)).astype(np.int64)
    plan = compute_layer_route(cu(ids), cu(parts), 1, CSRReplicaTable(cu(indptr), cu(ranks), cu(locs)), num_parts,
                               max_replicas_per_node=copies)
    ref = O.compute_layer_route(ids, np.arange(len(ids)), parts, 1, indptr, ranks, locs, num_parts)
    for a, b in zip((plan.send_ranks, plan.send_sizes, plan.send_indices, plan.send_remote_indices), ref):
        assert np.array_equal(npy(a), b)


@pytest.mark.parametrize("rank", [0, 3])
@pytest.mark.parametrize("copies", [255, 256, 257, 1000])
def test_route_plan_whose_ranks_fill_their_part_of_a_scan(copies, rank):
    """256 rows of one CTA with all copies on one rank: 65,280 places of a field of 16 bits, and more than it holds."""
    from starrygl.cache.cache_route import compute_layer_route
    from starrygl.cache.replica_table import CSRReplicaTable
    nodes = 600
    ids, parts = np.arange(nodes), np.ones(nodes, np.int64)
    indptr = np.concatenate([[0], np.cumsum(np.full(nodes, copies))]).astype(np.int64)
    ranks = np.full(indptr[-1], rank, np.int64)
    ranks[indptr[255]:indptr[256]:5] = 2                       # (the field behind the one that is full, or before it)
    ranks[indptr[255] + 1] = 4
    locs = np.arange(indptr[-1], dtype=np.int64)
    plan = compute_layer_route(cu(ids), cu(parts), 1, CSRReplicaTable(cu(indptr), cu(ranks), cu(locs)), 5, max_replicas_per_node=copies)
    ref = O.compute_layer_route(ids, np.arange(nodes), parts, 1, indptr, ranks, locs, 5)
    for a, b in zip((plan.send_ranks, plan.send_sizes, plan.send_indices, plan.send_remote_indices), ref):
        assert np.array_equal(npy(a), b)


def test_route_plan_of_more_entries_than_32_bits_count():
    """Every second node's copies are the same 2^20 table entries: 2^31 + 2^20 places in a plan with room for 1,000 of each rank's."""
    from starrygl import ops
    copies, rows, cap = 1 << 20, 2 * 2049, 1000
    indptr = torch.arange(rows + 1, device="cuda") % 2 * copies
    ranks = (torch.arange(copies, device="cuda") % 4 == 0).long() + 1                  # three quarters on rank 1, the others on rank 2
    locs = torch.arange(copies, device="cuda")
    st = ops.StatusWord(torch.device("cuda"))
    out_ranks, out_rows, out_locs, sizes, total = ops.plan_route(torch.arange(rows, device="cuda"), torch.zeros(rows, dtype=torch.int64, device="cuda"),
                                                                 0, indptr, ranks, locs, 3, cap, status=st)
    assert int(total) == 2049 * copies > 2 ** 31 and sizes.tolist() == [0, 2049 * copies // 4 * 3, 2049 * copies // 4]
    assert torch.equal(out_ranks, torch.ones_like(out_ranks)) and not out_rows.any()
    assert torch.equal(out_locs, locs[ranks == 1][:cap])
    with pytest.raises(Exception, match="capacity"):
        st.check("plan")


@pytest.mark.parametrize("fanouts", [[3], [10, 10], [4, 3, 2]])
@pytest.mark.parametrize("roots", [1, 700, 5000])
def test_layout_of_a_batch_next_to_its_last_merge(fanouts, roots):
    from starrygl import ops
    from starrygl.graph.batch import build_batch, build_batch_async
    rng = np.random.default_rng(roots)
    n, m = 3000, 40000
    src, dst, ts = rng.integers(0, n, m), rng.integers(0, n, m), np.sort(rng.integers(0, 10 ** 6, m))
    g = ops.tcsr_build(cu(src), cu(dst), cu(ts), None, n)
    pick = rng.integers(0, m, roots)
    for early in (False, True):                                # (queries before any event: hops without edges)
        q, t = cu(src[pick]), cu(np.zeros(roots, np.int64) if early else ts[pick])
        a, b = build_batch(g, q, t, fanouts, "recent"), build_batch_async(g, q, t, fanouts, "recent").finish()
        assert len(a) == len(b)
        for x, y in zip(a, b):
            assert list(x) == list(y)
            for k in x:
                assert x[k].dtype == y[k].dtype and torch.equal(x[k], y[k]), k


@pytest.mark.parametrize("fanouts", [[], [3], [4, 2]])
@pytest.mark.parametrize("roots", [0, 500])
@pytest.mark.parametrize("captured", [False, True])
def test_early_counts_come_with_every_batch(fanouts, roots, captured):
    """Also where the batch has no last merge, and where its kernels are captured instead of collected into a launch graph."""
    from starrygl import ops
    from starrygl.graph.batch import _enqueue
    rng = np.random.default_rng(roots)
    n, m = 300, 4000
    src, dst, ts = rng.integers(0, n, m), rng.integers(0, n, m), np.sort(rng.integers(0, 10 ** 6, m))
    g = ops.tcsr_build(cu(src), cu(dst), cu(ts), None, n)
    pick = rng.integers(0, m, roots)
    q, t = cu(src[pick]), cu(ts[pick])
    words, last = torch.zeros(64, dtype=torch.int64).pin_memory(), 1 + 2 * len(fanouts)

    def call():
        return _enqueue(g, q, t, fanouts, "recent", g.ts_min, g.ts_max, False, -1, 0, None, None, words.data_ptr(), early=words[32:].data_ptr())
    kept = call()
    if captured:
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            kept = call()
        words.fill_(-1)
        graph.replay()
    torch.cuda.synchronize()
    all_counts, early = words[:last + 2].tolist(), words[32:33 + last].tolist()
    assert all_counts[last:] == [0, 1] and early[last] == 1 and kept.n == roots
    known = last if not fanouts else last - 1
    assert early[:known] == all_counts[:known] and (roots == 0 or all_counts[0] > 0)
