"""Search index of the T-CSR at the edges of its kernel: entries of a CTA (256, or 1,024 from 1,212,416 entries on), rows without edges,
rows longer than a CTA's entries, a single row."""
import numpy as np
import pytest
import torch

from starrygl import ops

pytestmark = pytest.mark.gpu


def expected(indptr, ts, length):
    """fence[(s >> 5) + r + j] = time of the last edge of block j of row r; -1 where no row owns the entry."""
    s, e = indptr[:-1], indptr[1:]
    blocks = (e - s + 31) >> 5
    row = np.repeat(np.arange(len(s)), blocks)
    j = np.arange(len(row)) - np.repeat(np.cumsum(blocks) - blocks, blocks)
    out = np.full(length, -1, dtype=np.int64)
    out[(s[row] >> 5) + row + j] = ts[np.minimum(s[row] + 32 * j + 31, e[row] - 1)]
    return out


@pytest.mark.parametrize("nodes,edges,hub", [(1, 1, 0), (1, 70_000, 0), (2, 33, 33), (255, 1000, 0), (256, 31, 0), (257, 40_000, 39_000),
                                             (1023, 300_000, 299_000), (5000, 160_000, 9000), (1_212_415 - 3125, 100_000, 0),
                                             (1_212_416 - 3125, 100_000, 50_000), (1_300_001, 2_000_000, 1_500_000)])
def test_fence_of_every_row(nodes, edges, hub):
    rng = np.random.default_rng(nodes + edges)
    deg = np.bincount(rng.integers(0, nodes, edges - hub), minlength=nodes)
    deg[nodes // 2] += hub
    indptr = np.concatenate([[0], np.cumsum(deg)])
    ts = rng.integers(0, 1 << 40, edges)
    L = ops._C.lib()
    length = int(L.sgl_tcsr_fence_len(nodes, edges))
    d_ptr, d_ts = torch.from_numpy(indptr).cuda(), torch.from_numpy(ts).cuda()
    fence = torch.full((length,), -1, dtype=torch.int64, device="cuda")
    ops._C.check(L.sgl_tcsr_fence(d_ptr.data_ptr(), d_ts.data_ptr(), nodes, edges, fence.data_ptr(), ops._C.stream_ptr()))
    assert np.array_equal(fence.cpu().numpy(), expected(indptr, ts, length))
