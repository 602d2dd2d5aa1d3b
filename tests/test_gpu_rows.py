"""Row scatter: what is out of range or not stored here among rows that are in order, times and maps with them."""
import pytest
import torch

from starrygl import _C, ops

pytestmark = pytest.mark.gpu


def setup(dim, rows, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    table = torch.randn(rows, dim, device="cuda", generator=gen)
    ts = torch.rand(rows, device="cuda", generator=gen)
    return table, ts, torch.randperm(rows, device="cuda", generator=gen)[:n].contiguous(), gen


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
