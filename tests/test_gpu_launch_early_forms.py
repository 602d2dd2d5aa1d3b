"""Kernels that are set up while the one before them still runs, in the forms that a chain of plain gathers and scatters does not reach:
rows in 16-byte pieces (multiples of 16 bytes below 256, and longer ones asked for so), and index, map and count that the kernel just
before has written."""
import pytest
import torch

from starrygl import ops

pytestmark = pytest.mark.gpu
ROWS, N, ROUNDS = 40_001, 8_000, 12


def data(dim):
    gen = torch.Generator(device="cuda").manual_seed(dim)
    table = torch.randn(ROWS, dim, device="cuda", generator=gen)
    ts = torch.rand(ROWS, device="cuda", generator=gen)
    places = (torch.randperm(ROWS // 4 - 1, device="cuda", generator=gen)[:N] * 4).contiguous()     # (places of a round do not meet)
    return table, ts, places


def run(chain, captured, *state):
    if not captured:
        return chain(*state, ROUNDS)
    keep = [x.clone() for x in state]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain(*state, 1)
    torch.cuda.current_stream().wait_stream(side)
    for a, b in zip(state, keep):
        a.copy_(b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(*state, ROUNDS)
    graph.replay()


@pytest.mark.parametrize("dim,mode", [(4, "auto"), (20, "auto"), (60, "auto"), (100, "vec"), (3, "auto"), (186, "auto"), (128, "auto")])
@pytest.mark.parametrize("captured", [False, True])
def test_chain_of_rows(dim, mode, captured):
    table, ts, idx = data(dim)
    want, want_ts, at = table.clone(), ts.clone(), idx.clone()
    for _ in range(ROUNDS):
        want[at + 1], want_ts[at + 1] = want[at], want_ts[at]
        at = (at + 2) % (ROWS - 1)

    def chain(table, ts, idx, rounds):
        for _ in range(rounds):
            rows, t = ops.gather_rows(table, idx, ts_table=ts, mode=mode)
            ops.scatter_rows(table, idx + 1, rows, ts_table=ts, ts=t)
            idx.add_(2).remainder_(ROWS - 1)
    run(chain, captured, table, ts, idx)
    assert torch.equal(table, want) and torch.equal(ts, want_ts)


@pytest.mark.parametrize("dim,mode", [(4, "auto"), (20, "auto"), (3, "auto"), (128, "auto"), (100, "vec")])
@pytest.mark.parametrize("captured", [False, True])
def test_map_and_count_written_just_before(dim, mode, captured):
    """Ids go through a map that moves on every round, and only the first so many of them count, a number that changes every round."""
    table, ts, place = data(dim)
    ids = torch.randperm(N, device="cuda")
    to = torch.empty(N, dtype=torch.int64, device="cuda")
    to[:] = place
    n = torch.tensor([N], device="cuda")
    want, want_ts, m, count = table.clone(), ts.clone(), to.clone(), N
    for _ in range(ROUNDS):
        count -= 517
        at = m[ids[:count]]
        want[at + 1], want_ts[at + 1] = want[at], want_ts[at]
        m = (m + 2) % (ROWS - 1)

    def chain(table, ts, to, n, rounds):
        out = torch.empty(N, dim, device="cuda")
        for _ in range(rounds):
            n.sub_(517)
            _, t = ops.gather_rows(table, ids, map=to, d_n=n, ts_table=ts, mode=mode, out=out)
            to.add_(1)
            ops.scatter_rows(table, ids, out, map=to, d_n=n, ts_table=ts, ts=t)
            to.add_(1).remainder_(ROWS - 1)
    run(chain, captured, table, ts, to, n)
    assert torch.equal(table, want) and torch.equal(ts, want_ts)
