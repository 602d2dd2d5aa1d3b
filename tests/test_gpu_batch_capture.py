"""A whole batch with all its host words, captured on a stream and a second one: everything is joined into the first, and a replay writes
what a plain call writes."""
import ctypes as C

import pytest
import torch

from starrygl import _C, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fanouts", [[6], [5, 4], [4, 3, 2]])
@pytest.mark.parametrize("two", [False, True])
def test_captured_ready_word(fanouts, two):
    gen = torch.Generator(device="cuda").manual_seed(2)
    m, nodes, hops, n = 50_000, 3000, len(fanouts), 900
    src, dst = (torch.randint(0, nodes, (m,), device="cuda", generator=gen) for _ in range(2))
    ts = torch.randint(0, 1 << 20, (m,), device="cuda", generator=gen).sort().values
    g = ops.tcsr_build(src, dst, ts, torch.arange(m, device="cuda"), nodes)
    roots, times = src[m - n:].contiguous(), ts[m - n:].contiguous()
    L, k = _C.lib(), 3 + 14 * hops
    fan, size = (C.c_int32 * hops)(*fanouts), (C.c_int64 * k)()
    words = int(L.sgl_build_batch_layout(n, fan, hops, size))
    at = (C.c_int64 * k)(*[sum(size[:s]) for s in range(k)])
    ws = torch.empty(L.sgl_build_batch_ws_bytes(n, fan, hops), dtype=torch.uint8, device="cuda")
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    counts = 1 + 2 * hops

    def call(out, meta, p):
        _C.check(L.sgl_build_batch_ready(
            g.indptr.data_ptr(), g.nbr.data_ptr(), g.ts.data_ptr(), g.eid.data_ptr(), g.fence.data_ptr(), nodes, roots.data_ptr(), times.data_ptr(), n,
            fan, hops, 1, 0, -1, 5, 12, 20, 0, at, out.data_ptr(), 0, meta.data_ptr(), None, p, p + 8 * 20, p + 8 * 40, ws.data_ptr(), ws.numel(),
            side.cuda_stream if two else None, main.cuda_stream))

    def fresh():
        return (torch.zeros(words, dtype=torch.int64, device="cuda"), torch.zeros(2 + 2 * hops, dtype=torch.int64, device="cuda"),
                torch.full((64,), -1, dtype=torch.int64).pin_memory())
    want, want_meta, want_host = fresh()
    out, meta, host = fresh()
    torch.cuda.synchronize()
    call(want, want_meta, want_host.data_ptr())
    torch.cuda.synchronize()
    graph = C.c_void_p()
    _C.check(L.sgl_graph_capture_begin(main.cuda_stream))
    call(out, meta, host.data_ptr())
    _C.check(L.sgl_graph_capture_end(main.cuda_stream, C.byref(graph)))
    try:
        for _ in range(3):
            out.zero_(), meta.zero_()
            torch.cuda.synchronize()
            _C.check(L.sgl_graph_launch(graph, None, None, 0, main.cuda_stream))
            torch.cuda.synchronize()
            assert torch.equal(meta, want_meta) and torch.equal(host[:counts + 2], want_host[:counts + 2]) and host[40] == host[20 + counts] == 1
            c = want_meta.tolist()
            cuts = [(0, c[0]), (1, c[0]), (2, n)]
            for l in range(hops):
                b, e, u, rows = 3 + 14 * l, c[1 + 2 * l], c[2 + 2 * l], c[2 * l]
                cuts += [(b, e), (b + 2, e), (b + 4, e), (b + 6, u), (b + 7, u), (b + 8, e)]
                cuts += [(b + 9, rows + 1), (b + 10, e), (b + 11, e), (b + 13, e)] if l else []
            assert all(torch.equal(out[at[s]:at[s] + x], want[at[s]:at[s] + x]) for s, x in cuts)
    finally:
        L.sgl_graph_destroy(graph)
