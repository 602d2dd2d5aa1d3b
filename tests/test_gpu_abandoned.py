"""Slots and batches that fail between their launches and their end: nothing of them is running when the error arrives, and what the thread
builds next, smaller and larger, is right."""
import numpy as np
import pytest
import torch

from starrygl.graph import batch
from starrygl.graph.batch import build_batch

from test_gpu_slot_copies import M, check, make, slot

pytestmark = pytest.mark.gpu


class Stop(Exception):
    pass


@pytest.mark.parametrize("where", ["plan", "copies", "first copy", "second copy"])
def test_slot(monkeypatch, where):
    data, b = make(4)
    check(data, b, M // 2, M // 2 + 50, [10, 10], "recent")
    calls = []

    def fail(*a, **k):
        calls.append(a)
        if where == "second copy" and len(calls) == 1:
            return real(*a, **k)
        raise Stop
    name = {"plan": "_plan", "copies": "_copies"}.get(where, "_export")
    real = getattr(b, name)
    monkeypatch.setattr(b, name, fail, raising=False)
    with pytest.raises(Stop):
        slot(data, b, M // 4, M // 4 + 9000, [20, 20], "uniform")
    assert torch.cuda.current_stream().query()
    monkeypatch.undo()
    for n in (1, 40, 3000):
        check(data, b, M // 2, M // 2 + n, [10, 10], "recent")


def test_batch(monkeypatch):
    data, b = make(1)
    pick = lambda a, e: (torch.from_numpy(np.concatenate([data["src"][a:e], data["dst"][a:e]])).cuda(),
                         torch.from_numpy(np.concatenate([data["ts"][a:e]] * 2)).cuda())
    small, large = pick(M // 2, M // 2 + 40), pick(M // 4, M // 4 + 9000)
    want = build_batch(b.g, *small, [10, 10])

    def fail(self, host):
        raise Stop
    monkeypatch.setattr(batch.DeviceBatch, "_trim_but_last", fail)
    with pytest.raises(Stop):
        build_batch(b.g, *large, [20, 20], "uniform")
    assert torch.cuda.current_stream().query()
    monkeypatch.undo()
    for d, w in zip(build_batch(b.g, *small, [10, 10]), want):
        assert list(d) == list(w) and all(torch.equal(d[k], w[k]) for k in w)
