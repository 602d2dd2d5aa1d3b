"""Batches are submitted in two parts: a thread keeps graphs for as many streams (or kinds of batches) as for calls that are submitted whole."""
import threading

import pytest
import torch

from starrygl import _C, ops
from starrygl.graph.batch import build_batch

pytestmark = pytest.mark.gpu


def test_batches_on_many_streams_keep_their_graphs():
    gen = torch.Generator(device="cuda").manual_seed(1)
    m, n = 40_000, 2000
    src, dst = (torch.randint(0, n, (m,), device="cuda", generator=gen) for _ in range(2))
    ts = torch.randint(0, 10 ** 6, (m,), device="cuda", generator=gen).sort().values
    g = ops.tcsr_build(src, dst, ts, torch.arange(m, device="cuda"), n)
    roots, times = src[-1000:].contiguous(), ts[-1000:].contiguous()
    want = build_batch(g, roots, times, [10])
    torch.cuda.synchronize()
    held, wrong = [], []

    def work():
        streams = [torch.cuda.Stream() for _ in range(24)]
        for r in range(4):
            for s in streams:
                with torch.cuda.stream(s):
                    got = build_batch(g, roots, times, [10])
                    wrong.extend(k for d, w in zip(got, want) for k in w if not torch.equal(d[k], w[k]))
            held.append(_C.lib().sgl_launch_graphs())
    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not wrong
    assert held == [0, 24, 24, 24]
