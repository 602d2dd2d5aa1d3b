"""Slots whose arrays reach the host in two parts, the first next to the merge of the last list: against the same batch built on the device.
One hop (nothing but the last list is merged), several, more counts than the result words hold apart, hops without edges, many threads."""
import threading

import numpy as np
import pytest
import torch

from starrygl.cache.replica_table import CSRReplicaTable
from starrygl.graph.batch import build_batch
from starrygl.graph.materialize import MaterializedMultiLayerBuilder

pytestmark = pytest.mark.gpu
N, M = 3000, 60_000


def make(parts, seed=0):
    rng = np.random.default_rng(seed)
    data = dict(src=rng.integers(0, N, M), dst=rng.integers(0, N, M), ts=np.sort(rng.integers(0, 10 ** 6, M)), eid=np.arange(M))
    if parts == 1:
        return data, MaterializedMultiLayerBuilder(data, N, None, None, 0, 1)
    owner = torch.from_numpy(rng.integers(0, parts, N))
    held = torch.from_numpy(rng.random((N, parts)) < 0.2)
    held[torch.arange(N), owner] = True
    ptr = torch.zeros(N + 1, dtype=torch.int64)
    ptr[1:] = held.sum(1).cumsum(0)
    slot, rank = held.long().cumsum(0) - 1, torch.arange(parts).expand(N, parts)
    table = CSRReplicaTable(ptr.cuda(), rank[held].contiguous().cuda(), slot[held].contiguous().cuda())
    return data, MaterializedMultiLayerBuilder(data, N, owner.cuda(), table, 0, parts)


def slot(data, b, a, e, fanouts, policy):
    task = ("link", (data["src"][a:e], data["dst"][a:e], data["ts"][a:e], np.zeros(e - a), data["eid"][a:e]))
    layers = {"meta": {"graph_type": "c", "end_offset": 0}, "layer": [{"type": policy, "fanout": k} for k in fanouts]}
    return b.build_aligned_batch(task, None, layers, seed=1)


def check(data, b, a, e, fanouts, policy):
    got = slot(data, b, a, e, fanouts, policy)
    roots = torch.from_numpy(np.concatenate([data["src"][a:e], data["dst"][a:e]])).cuda()
    times = torch.from_numpy(np.concatenate([data["ts"][a:e]] * 2)).cuda()
    want = build_batch(b.g, roots, times, fanouts, policy, seed=1)
    assert len(got) == len(want)
    for d, w in zip(got, want):
        assert list(w) == [k for k in d if k in w]
        for k in w:
            assert torch.equal(d[k], w[k].cpu()), k


@pytest.mark.parametrize("policy", ["recent", "uniform"])
@pytest.mark.parametrize("parts,fanouts", [(1, [10]), (4, [10]), (1, [5, 5]), (4, [10, 10]), (2, [4, 3, 2]), (30, [2] * 8), (2, [])])
def test_both_parts(parts, fanouts, policy):
    data, b = make(parts)
    for a, e in ((M // 2, M // 2 + 1), (M // 2, M // 2 + 700), (M - 40, M)):
        check(data, b, a, e, fanouts, policy)


def test_hops_without_edges():
    data, b = make(4)
    for a, e in ((0, 1), (0, 3), (3, 60)):
        check(data, b, a, e, [10, 10], "recent")


def test_threads_side_by_side():
    data, b = make(4)
    wrong = []

    def work(i):
        try:
            torch.cuda.set_device(0)
            with torch.cuda.stream(torch.cuda.Stream()):
                for r in range(4):
                    a = M // 4 + 4000 * i + 900 * r
                    check(data, b, a, a + 300 + 100 * i, [10, 5], "recent")
        except BaseException as e:
            wrong.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if wrong:
        raise wrong[0]
