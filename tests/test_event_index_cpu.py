"""Host-known bounds of a time window's events, from every 256th timestamp: no object per entry is made for them, and they hold the window."""
import numpy as np
import pytest
import torch

from starrygl.lib.libstarrygl_comm import CUDAGraph


def graph(ts):
    g = CUDAGraph.__new__(CUDAGraph)
    g.ev, g.stream, g._ev_index, g._closed, g._results = (None, torch.from_numpy(ts), None), None, None, True, ()
    return g


@pytest.mark.parametrize("m,span", [(1, 1), (255, 10), (256, 3), (257, 10 ** 6), (5000, 40), (100_000, 10 ** 9)])
def test_bounds_hold_the_window(m, span):
    rng = np.random.default_rng(m)
    ts = np.sort(rng.integers(-span, span + 1, m))
    g = graph(ts)
    for t0 in (-2 ** 63, -span - 1, 0, 5, span, span + 1, 2 ** 63 - 1, *rng.integers(-span, span + 1, 20).tolist()):
        for t1 in (t0, t0 + 1, t0 + span // 3, span + 5):
            first, most = g._window(t0, t1)
            lo, hi = np.searchsorted(ts, [max(t0, -2 ** 62), min(max(t1, -2 ** 62), 2 ** 62)])
            assert 0 <= first < m and 1 <= most <= m - first
            assert hi <= lo or (first <= lo and hi <= first + most)
            assert most <= max(hi - lo, 0) + 512
    assert not isinstance(g._ev_index, (list, tuple)) and len(g._ev_index) == (m + 255) // 256
