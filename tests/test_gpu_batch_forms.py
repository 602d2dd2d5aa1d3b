"""The C entry points of a whole batch leave the same arrays: in one arena, with a place for every section, with early counts, with the word
that says that all but the last list may be read."""
import ctypes as C

import pytest
import torch

from starrygl import _C, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fanouts", [[7], [5, 4], [4, 3, 2], []])
@pytest.mark.parametrize("n", [0, 1, 700])
def test_forms_agree(fanouts, n):
    gen = torch.Generator(device="cuda").manual_seed(n)
    m, nodes, hops = 50_000, 3000, len(fanouts)
    src, dst = (torch.randint(0, nodes, (m,), device="cuda", generator=gen) for _ in range(2))
    ts = torch.randint(0, 1 << 20, (m,), device="cuda", generator=gen).sort().values
    g = ops.tcsr_build(src, dst, ts, torch.arange(m, device="cuda"), nodes)
    roots, times = src[m - n:].contiguous(), ts[m - n:].contiguous()
    L, k = _C.lib(), 3 + 14 * hops
    fan, size = (C.c_int32 * max(hops, 1))(*fanouts), (C.c_int64 * k)()
    words = L.sgl_build_batch_layout(n, fan, hops, size)
    at = (C.c_int64 * k)(*[sum(size[:s]) for s in range(k)])
    ws = torch.empty(max(L.sgl_build_batch_ws_bytes(n, fan, hops), 256), dtype=torch.uint8, device="cuda")
    head = [g.indptr.data_ptr(), g.nbr.data_ptr(), g.ts.data_ptr(), g.eid.data_ptr(), g.fence.data_ptr(), nodes, roots.data_ptr(), times.data_ptr(), n,
            fan, hops, 1, 0, -1, 5, 12, 20, 0]
    counts = 1 + 2 * hops
    results = []
    for form in ("", "_at", "_staged", "_ready"):
        out = torch.zeros(max(int(words), 1), dtype=torch.int64, device="cuda")
        meta = torch.zeros(2 + 2 * hops, dtype=torch.int64, device="cuda")
        host = torch.full((64,), -1, dtype=torch.int64).pin_memory()
        p = host.data_ptr()
        early = {"_staged": [p + 8 * 20], "_ready": [p + 8 * 20, p + 8 * 40]}.get(form, [])
        places = [] if form == "" else [at]
        base = [out.data_ptr()] if form == "" else [out.data_ptr(), 0]
        sp = _C.stream_ptr()
        _C.check(getattr(L, "sgl_build_batch" + form)(*head, *places, *base, meta.data_ptr(), None, p, *early, ws.data_ptr(), ws.numel(), None, sp))
        for flag in [p + 8 * (counts + 1)] + ([p + 8 * (20 + counts)] if early else []) + ([p + 8 * 40] if form == "_ready" else []):
            _C.check(L.sgl_wait_word(flag, 1, sp))
        torch.cuda.synchronize()
        assert host[:counts + 1].tolist() == meta.tolist() and host[counts].item() == 0
        if early:
            known = counts - 1 if hops else counts                 # all but the last list's length
            assert host[20:20 + known].tolist() == meta[:known].tolist()
        # every section up to its count
        c = meta.tolist()
        kept = [out[at[0]:at[0] + c[0]], out[at[1]:at[1] + c[0]], out[at[2]:at[2] + n]]
        for l in range(hops):
            b, e, u, rows = 3 + 14 * l, c[1 + 2 * l], c[2 + 2 * l], c[2 * l]
            cut = lambda s, k: out[at[b + s]:at[b + s] + k]
            kept += [cut(0, e), cut(2, e), cut(4, e), cut(6, u), cut(7, u), cut(8, e)]
            if l:
                kept += [cut(9, rows + 1), cut(10, e), cut(11, e), cut(13, e)]
        results.append((c, [x.clone() for x in kept if n]))
    for c, kept in results[1:]:
        assert c == results[0][0] and all(torch.equal(a, b) for a, b in zip(kept, results[0][1]))
