"""Slot files written by the GPU builder (``starrygl.graph.materialize``) against the files the reference's
``build_aligned_batch`` wrote for the same partitions and tasks (golden ``slots.npz``): same keys, same tensors, same
per-layer route plans (inside a destination-rank segment the reference's order comes from an unstable argsort, so
segments are compared as multisets)."""
import os

import numpy as np
import pytest
import torch

from gpu_util import load
from test_oracle_golden import LAYER_KEYS, same_plan_up_to_segment_order, slot_cases

pytestmark = pytest.mark.gpu


def test_slot_files_match_the_reference(tmp_path):
    from starrygl.cache.replica_table import CSRReplicaTable
    from starrygl.graph.materialize import MaterializedMultiLayerBuilder
    builders = {}
    for z, c, pid, roots, rts in slot_cases():
        if pid not in builders:
            rt = CSRReplicaTable(torch.from_numpy(z["rt_indptr"]), torch.from_numpy(z["rt_ranks"]), torch.from_numpy(z["rt_locs"]))
            builders[pid] = MaterializedMultiLayerBuilder({k: z[k] for k in ("src", "dst", "ts", "eid")}, int(z["N"]),
                                                          torch.from_numpy(z["node_parts"]), rt, pid, int(z["P"]))
        pick = z[f"c{c}_pick"]
        kind = str(z[f"c{c}_kind"])
        if kind == "link":
            task = ('link', (z["src"][pick], z["dst"][pick], z["ts"][pick], np.ones(len(pick), np.int64), z["eid"][pick]))
        else:
            task = ('node', (z["dst"][pick], z["ts"][pick], np.zeros(len(pick), np.int64)))
        cfg = {'meta': {'start_offset': -1, 'end_offset': int(z[f"c{c}_end_offset"]), 'graph_type': 'c'},
               'layer': [{'type': 'recent', 'fanout': int(f)} for f in z[f"c{c}_fanouts"]]}
        path = os.path.join(tmp_path, f"slot_{c:04d}_sub_{pid:04d}.pt")
        builders[pid].build_aligned_batch(task, path, cfg, 1, None, None)
        data = torch.load(path, weights_only=False)          # what a loader of the reference would read
        tag = f"c{c}_p{pid}"
        assert len(data) == int(z[f"{tag}_num_layers"])
        ref_keys = {f[len(tag) + 4:] for f in z.files if f.startswith(f"{tag}_L0_")}
        assert ref_keys <= set(data[0].keys()) and "comm_plan" in data[0], (tag, ref_keys - set(data[0].keys()))
        for k in ref_keys:
            v = data[0][k]
            assert not (torch.is_tensor(v) and v.is_cuda)
            assert np.array_equal(np.asarray(v), z[f"{tag}_L0_{k}"]), (tag, k)
        for i in range(1, len(data)):
            assert set(data[i].keys()) == set(LAYER_KEYS)
            for k in LAYER_KEYS:
                a, r = data[i][k].numpy(), z[f"{tag}_L{i}_{k}"]
                assert a.dtype == r.dtype and np.array_equal(a, r), (tag, i, k)
        plans = data[0]["comm_plan"]
        assert len(plans) == int(z[f"{tag}_num_plans"])
        for i, pl in enumerate(plans):
            got = None if pl is None else (pl.send_ranks.numpy(), pl.send_sizes.numpy(), pl.send_indices.numpy(),
                                           pl.send_remote_indices.numpy())
            assert same_plan_up_to_segment_order(got, z, f"{tag}_plan{i}"), (tag, i)


def test_unsupported_policies_raise():
    from starrygl.graph.materialize import MaterializedMultiLayerBuilder
    e = np.arange(4, dtype=np.int64)
    b = MaterializedMultiLayerBuilder({'src': e, 'dst': e[::-1].copy(), 'ts': e}, 4, None, None, 0, 1)
    task = ('node', (e, e + 10, e))
    for cfg in ({'meta': {'graph_type': 'd'}, 'layer': [{'type': 'recent', 'fanout': 2}]},
                {'meta': {}, 'layer': [{'type': 'cluster', 'fanout': 2}]},
                {'meta': {'end_offset': 5}, 'layer': [{'type': 'recent', 'fanout': 2}]}):
        with pytest.raises(NotImplementedError):
            b.build_aligned_batch(task, None, cfg)
    out = b.build_aligned_batch(task, None, {'meta': {}, 'layer': [{'type': 'uniform', 'fanout': 2}]}, seed=3)
    assert out[0]["comm_plan"] == [None, None] and out[1]["indptr"].numel() == out[0]["gids"].numel() + 1


def test_one_builder_in_two_threads():
    """Slots built side by side with one builder, each thread on a stream of its own, are those of one thread."""
    import threading
    from starrygl.graph.materialize import MaterializedMultiLayerBuilder
    rng = np.random.default_rng(0)
    n, m = 5000, 100000
    z = {k: rng.integers(0, n, m).astype(np.int64) for k in ("src", "dst")}
    z["ts"] = np.sort(rng.integers(0, 10 ** 6, m)).astype(np.int64)
    b = MaterializedMultiLayerBuilder(z, n, None, None, 0, 1)
    cfg = {'meta': {}, 'layer': [{'type': 'recent', 'fanout': 5}]}

    def slot(i):
        at = slice(50000 + 100 * i, 50000 + 100 * i + 3000)
        return b.build_aligned_batch(('node', (z["src"][at], z["ts"][at], np.zeros(3000))), None, cfg)
    want = [slot(i) for i in range(100)]
    wrong = []

    def work(first):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(first, 100, 2):
                got = slot(i)
                if not all(torch.equal(got[l][k], want[i][l][k]) for l in range(2) for k in ("gids", "ts")):
                    wrong.append(i)
    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong


@pytest.mark.parametrize("events", [500, 60000])
def test_one_tensor_of_a_slot_stands_for_itself(events, tmp_path):
    """Saved alone it is a file of its own size; in a large slot it holds no other's memory.  Both forms of the copy."""
    from starrygl.graph.materialize import MaterializedMultiLayerBuilder
    rng = np.random.default_rng(0)
    n, m = 50000, 400000
    z = {k: rng.integers(0, n, m).astype(np.int64) for k in ("src", "dst")}
    z["ts"] = np.sort(rng.integers(0, 10 ** 6, m)).astype(np.int64)
    b = MaterializedMultiLayerBuilder(z, n, None, None, 0, 1)
    at = slice(300000, 300000 + events)
    out = b.build_aligned_batch(('node', (z["src"][at], z["ts"][at], np.zeros(events))), None,
                                {'meta': {}, 'layer': [{'type': 'recent', 'fanout': 5}] * 2})
    from oracle import oracle_np as O
    csr = O.tcsr_build(z["dst"], z["src"], z["ts"], np.arange(m), n)[:4]
    ref = O.build_batch(*csr, z["src"][at], z["ts"][at], [5, 5])
    total = 0
    for d, r in zip(out, ref):
        for k in r:
            assert np.array_equal(d[k].numpy(), r[k]), k
            assert d[k].untyped_storage().nbytes() == d[k].numel() * d[k].element_size(), k
            total += d[k].untyped_storage().nbytes()
    assert (total > 32 << 20) == (events == 60000)
    path = os.path.join(tmp_path, "one.pt")
    torch.save(out[1]["indptr"], path)
    assert os.path.getsize(path) < out[1]["indptr"].numel() * 8 + 4096


@pytest.mark.parametrize("hops", [9, 10, 12])
def test_slots_of_many_hops(hops):
    from oracle import oracle_np as O
    from starrygl.cache.replica_table import CSRReplicaTable
    from starrygl.graph.materialize import MaterializedMultiLayerBuilder
    rng = np.random.default_rng(0)
    n, m, parts = 300, 40000, 3
    z = {k: rng.integers(0, n, m).astype(np.int64) for k in ("src", "dst")}
    z["ts"] = np.sort(rng.integers(0, 10 ** 6, m)).astype(np.int64)
    ranks = torch.arange(parts).repeat(n)                 # every node on every partition
    table = CSRReplicaTable(torch.arange(n + 1) * parts, ranks, torch.arange(n).repeat_interleave(parts))
    node_parts = torch.arange(n) % parts
    b = MaterializedMultiLayerBuilder(z, n, node_parts, table, 0, parts)
    roots, rts = rng.integers(0, n, 50).astype(np.int64), np.full(50, 10 ** 6 - 1, np.int64)
    out = b.build_aligned_batch(('node', (roots, rts, np.zeros(50))), None, {'meta': {}, 'layer': [{'type': 'recent', 'fanout': 1}] * hops})
    ref = O.build_batch(*O.tcsr_build(z["dst"], z["src"], z["ts"], np.arange(m), n)[:4], roots, rts, [1] * hops)
    assert len(out) == len(ref) == hops + 1 and len(out[0]["comm_plan"]) == hops + 1
    for d, r, p in zip(out, ref, out[0]["comm_plan"]):
        for k in r:
            assert np.array_equal(d[k].numpy(), r[k]), k
        gids = r["gids"]
        last = np.append(gids[1:] != gids[:-1], True) & (gids % parts == 0)
        assert np.array_equal(p.send_indices.numpy(), np.tile(last.nonzero()[0], 2)) and p.send_sizes.tolist() == [0, last.sum(), last.sum()]
