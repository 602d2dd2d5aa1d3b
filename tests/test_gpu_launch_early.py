"""Kernels that are set up while the one before them still runs: chains of gathers and scatters that each need all of what the last one
wrote, with nothing between them on the stream, after a torch kernel, and as a captured graph."""
import pytest
import torch

from starrygl import ops

pytestmark = pytest.mark.gpu


def chain(table, ts, idx, rounds):
    """Rows (and times) of idx go to the places next to them, and the places move on: every round reads what the last one wrote."""
    for _ in range(rounds):
        rows, t = ops.gather_rows(table, idx, ts_table=ts)
        ops.scatter_rows(table, idx + 1, rows, ts_table=ts, ts=t)
        rows, t = ops.gather_rows(table, idx + 1, ts_table=ts)
        ops.scatter_rows(table, idx, rows, ts_table=ts, ts=t)
        idx.add_(2).remainder_(table.shape[0] - 1)          # read by the next gather, written just before it


def reference(table, ts, idx, rounds):
    for _ in range(rounds):
        table[idx + 1], ts[idx + 1] = table[idx], ts[idx]
        idx = (idx + 2) % (table.shape[0] - 1)


@pytest.mark.parametrize("dim", [1, 3, 100, 128, 186])      # 4-byte pieces (1, 3, 186), the bulk copy
@pytest.mark.parametrize("captured", [False, True])
def test_each_round_sees_the_last_one(dim, captured):
    rows, n, rounds = 40_001, 8_000, 12
    gen = torch.Generator(device="cuda").manual_seed(dim)
    table = torch.randn(rows, dim, device="cuda", generator=gen)
    ts = torch.rand(rows, device="cuda", generator=gen)
    idx = (torch.randperm(rows // 4 - 1, device="cuda", generator=gen)[:n] * 4).contiguous()     # (places of a round do not meet)
    want, want_ts = table.clone(), ts.clone()
    reference(want, want_ts, idx.clone(), rounds)
    if captured:
        keep = table.clone(), ts.clone(), idx.clone()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            chain(table, ts, idx, 1)
        torch.cuda.current_stream().wait_stream(side)
        for a, b in zip((table, ts, idx), keep):
            a.copy_(b)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            chain(table, ts, idx, rounds)
        graph.replay()
    else:
        chain(table, ts, idx, rounds)
    assert torch.equal(table, want) and torch.equal(ts, want_ts)
