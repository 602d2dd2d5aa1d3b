"""A slot or batch that fails behind its launches waits for them before the error leaves it: the thread's next call uses the same result
words.  (The device side is a fake here; tests/test_gpu_abandoned.py runs the real one.)"""
import types

import pytest
import torch

from starrygl import _C
from starrygl.graph import batch, materialize


@pytest.fixture
def fakes(monkeypatch):
    log = []
    words = [0] * 512
    for i in (materialize._EARLY, materialize._EARLY + 1, materialize._EARLY + 2):
        words[i] = 3

    class DB:
        def addresses(self):
            return [0] * 64

        def _trim_but_last(self, counts):
            raise KeyboardInterrupt
    monkeypatch.setattr(_C, "host_words", lambda: (0, words))
    monkeypatch.setattr(_C, "host", lambda: types.SimpleNamespace(sgl_wait_word=lambda *a: log.append("wait")))
    monkeypatch.setattr(_C, "stream_ptr", lambda *a: 0)
    monkeypatch.setattr(_C, "current_stream", lambda *a: types.SimpleNamespace(synchronize=lambda: log.append("idle")))
    monkeypatch.setattr(torch._C, "_cuda_isCurrentStreamCapturing", lambda: False, raising=False)
    for m in (batch, materialize):
        monkeypatch.setattr(m, "_enqueue", lambda *a, **k: log.append("enqueued") or DB())
        monkeypatch.setattr(m, "_graph_range", lambda g, lo, hi: (lo, hi))
    return log


def builder(**kw):
    b = materialize.MaterializedMultiLayerBuilder.__new__(materialize.MaterializedMultiLayerBuilder)
    b.__dict__.update(dict(g=None, num_parts=1, rep_table=None, node_parts=None, device=torch.device("cpu")), **kw)
    return b


def refuse(*a, **k):
    raise _C.SglError("refused")


@pytest.mark.parametrize("where", ["plan", "early copies", "end"])
def test_slot(fakes, monkeypatch, where):
    b = builder()
    if where == "plan":
        b.num_parts, b.rep_table, b.node_parts, b._plan = 2, object(), object(), refuse
    elif where == "early copies":
        b._copies = refuse
    else:
        b._copies = lambda: types.SimpleNamespace(synchronize=lambda: fakes.append("copies idle"))
        monkeypatch.setattr(_C, "on_stream", lambda s: __import__("contextlib").nullcontext())
        b._export, b._finish = (lambda picks, ready=None: [None] * len(picks)), refuse
    roots = torch.arange(5)
    with pytest.raises(_C.SglError, match="refused"):
        b._build(roots, roots, (0, 4), [2], "recent", False, 0)
    assert fakes.index("idle") > fakes.index("enqueued")
    assert where != "end" or fakes[-1] == "copies idle"


def test_batch(fakes):
    g = types.SimpleNamespace(ts_min=0, ts_max=9)
    with pytest.raises(KeyboardInterrupt):
        batch.build_batch(g, torch.arange(5), torch.arange(5), [2])
    assert fakes == ["enqueued", "wait", "idle"]


def test_capturing_stream_is_left_alone(fakes, monkeypatch):
    monkeypatch.setattr(torch._C, "_cuda_isCurrentStreamCapturing", lambda: True)
    _C.abandon()
    assert fakes == []
