"""T-CSR builds by radix passes whose ids turn out to be wide while the digits are counted: the passes of that sort do nothing (so nothing is
left of it), and the build with positions follows.  One such id, ids in every warp, alone and with the search index."""
import numpy as np
import pytest
import torch

from starrygl import ops

from test_gpu_tcsr_ids import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1_212_417, 1_500_001, 4_000_003])
@pytest.mark.parametrize("kind", ["one", "every", "negative", "ordered"])
def test_wide_ids_in_the_middle(m, kind):
    rng = np.random.default_rng(m)
    nodes = 30_000
    key, nbr, ts, eid = rng.integers(0, nodes, m), rng.integers(0, nodes, m), rng.integers(0, 1 << 24, m), np.arange(m)
    mid = slice(m // 2 - 200_000, m // 2 + 200_000) if kind == "every" else m // 2
    if kind == "ordered":
        ts.sort()
    nbr[mid] = -5 if kind == "negative" else (1 << 40) + 7
    check(key, nbr, ts, eid, nodes)


def test_index_of_such_a_build_and_the_next_one():
    m, nodes = 2_000_000, 20_000
    gen = torch.Generator(device="cuda").manual_seed(3)
    key, nbr = (torch.randint(0, nodes, (m,), device="cuda", generator=gen) for _ in range(2))
    ts, eid = torch.randint(0, 1 << 24, (m,), device="cuda", generator=gen), torch.arange(m, device="cuda")
    narrow = ops.tcsr_build(key, nbr, ts, eid, nodes)
    eid[m // 2] = 1 << 33
    for _ in range(3):
        wide = ops.tcsr_build(key, nbr, ts, eid, nodes)
        again = ops.tcsr_build(key, nbr, ts, torch.arange(m, device="cuda"), nodes)
        for g in (wide, again):
            assert torch.equal(g.indptr, narrow.indptr) and torch.equal(g.ts, narrow.ts) and torch.equal(g.nbr, narrow.nbr)
            rows, j = narrow.indptr[:-1], (narrow.indptr[1:] - narrow.indptr[:-1] + 31) >> 5
            at = ((rows >> 5) + torch.arange(nodes, device="cuda")).repeat_interleave(j)
            at += torch.arange(at.numel(), device="cuda") - (j.cumsum(0) - j).repeat_interleave(j)
            assert torch.equal(g.fence[at], narrow.fence[at])
        assert torch.equal(again.eid, narrow.eid) and int((wide.eid == 1 << 33).sum()) == 1
