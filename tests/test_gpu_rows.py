"""Row gather and scatter: what is out of range or not stored here among pieces that are in order, times and maps with them."""
import pytest
import torch

from starrygl import _C, ops

pytestmark = pytest.mark.gpu


def setup(dim, rows, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    table = torch.randn(rows, dim, device="cuda", generator=gen)
    ts = torch.rand(rows, device="cuda", generator=gen)
    return table, ts, torch.randperm(rows, device="cuda", generator=gen)[:n].contiguous(), gen


@pytest.mark.parametrize("dim", [1, 3, 4, 20, 36, 386])         # 4- and 16-byte pieces (36: 144 bytes)
@pytest.mark.parametrize("mapped", [False, True])
def test_gather_around_bad_rows(dim, mapped):
    rows, n = 500_000, 301_000                                  # several pieces a thread, at 386 several rounds
    if dim == 386:
        rows, n = 60_000, 30_001
    table, ts, want, gen = setup(dim, rows, n, dim)
    to = torch.randperm(rows, device="cuda", generator=gen)
    idx = torch.argsort(to)[want].contiguous() if mapped else want.clone()
    idx[::7] = -1 - torch.arange(idx[::7].numel(), device="cuda") if not mapped else idx[::7]
    want = want.clone()
    if not mapped:
        want[::7] = rows - 1 - torch.arange(want[::7].numel(), device="cuda")       # (below 0: from the end)
    bad = torch.zeros(n, dtype=torch.bool, device="cuda")
    bad[5::1000] = True
    idx[5::1000], idx[5::2000] = rows, (-1 if mapped else -rows - 1)
    st = ops.StatusWord(table.device)
    out = torch.full((n, dim), -7.0, device="cuda")
    got, got_ts = ops.gather_rows(table, idx, map=to if mapped else None, ts_table=ts, out=out, mode="vec" if dim % 4 == 0 else "auto", status=st)
    assert got is out and torch.equal(out[~bad], table[want[~bad]]) and torch.equal(got_ts[~bad], ts[want[~bad]])
    assert bool((out[bad] == -7.0).all())                       # (left as they are)
    with pytest.raises(_C.SglError, match="row index out of range"):
        st.check()


@pytest.mark.parametrize("dim", [1, 3, 4, 36, 100, 186])
@pytest.mark.parametrize("mapped", [False, True])
def test_scatter_needs_no_source_without_a_destination(dim, mapped):
    rows, n, here = 400_000, 90_001, 50_003
    table, ts, place, gen = setup(dim, rows, here, dim)
    src, st = torch.randn(here, dim, device="cuda", generator=gen), torch.rand(here, device="cuda", generator=gen)
    idx = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    idx[:here] = place
    to = None
    if mapped:                                                  # entries behind `here` are known but not stored here
        to = torch.full((n,), -1, dtype=torch.int64, device="cuda")
        to[:here] = place
        idx = torch.arange(n, device="cuda")
    want, want_ts = table.clone(), ts.clone()
    want[place], want_ts[place] = src, st
    status = ops.StatusWord(table.device)
    ops.scatter_rows(table, idx, src, map=to, ts_table=ts, ts=st, status=status)
    assert torch.equal(table, want) and torch.equal(ts, want_ts)
    status.check()
    idx[3] = rows if not mapped else n
    ops.scatter_rows(table, idx, src, map=to, ts_table=ts, ts=st, status=status)
    assert torch.equal(table, want)
    with pytest.raises(_C.SglError, match="row index out of range"):
        status.check()
