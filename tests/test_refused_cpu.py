"""A batch or query whose hops cannot be built is refused before anything is launched (so these calls need no GPU), not behind its first list."""
import ctypes as C

import pytest

from starrygl import _C

PTR = 1 << 20                # (never followed: the calls are refused)


def batch(fanouts, policy=1, roots=1000, graph=PTR, id_bits=20, ts_bits=24, sections=None):
    L, k = _C.lib(), len(fanouts)
    fan = (C.c_int32 * k)(*fanouts)
    at = (C.c_int64 * (3 + 14 * k))(*(sections or range(1, 4 + 14 * k)))
    return L.sgl_build_batch_ready(graph, PTR, PTR, PTR, None, 1000, PTR, PTR, roots, fan, k, policy, 0, -1, 0, id_bits, ts_bits, 0, at,
                                   0 if sections else PTR, 0, PTR, None, None, None, None, PTR, 1 << 62, None, None)


@pytest.mark.parametrize("rc,text,kw", [
    (-5, "uniform fanout 513", dict(fanouts=[10, 513])),
    (-1, "unknown policy 7", dict(fanouts=[10], policy=7)),
    (-1, "null array", dict(fanouts=[10, 10], graph=None)),
    (-1, "null section", dict(fanouts=[10, 10], sections=[1, 2, 3] + [0] * 28)),
    (-5, "64-bit positions", dict(fanouts=[512, 512, 32], policy=0)),             # 8.6 x 10^9 edges
    (-5, "64-bit positions", dict(fanouts=[10], roots=390_451_573)),              # 11 x that: 2^32 + 7
    (-5, "64-bit positions", dict(fanouts=[512] * 8)),                            # (beyond 64 bits)
    (-5, "64-bit sort key", dict(fanouts=[10, 10], id_bits=0, ts_bits=60)),       # rows of the second CSC and times
])
def test_batch(rc, text, kw):
    assert batch(**kw) == rc, _C.lib().sgl_last_error()
    assert text in _C.lib().sgl_last_error().decode()


@pytest.mark.parametrize("rc,text,kw", [
    (-5, "uniform fanout 600", dict(fanout=600)),
    (-1, "unknown policy 3", dict(policy=3)),
    (-1, "fanout=0", dict(fanout=0)),
    (-1, "null array", dict(graph=None)),
    (-5, "64-bit position", dict(fanout=400, hops=3, policy=0)),
    (-5, "num_nodes too large", dict(nodes=(1 << 63) - 1)),
    (-1, "negative size", dict(nodes=-1)),
])
def test_query(rc, text, kw):
    a = dict(dict(fanout=10, hops=2, policy=1, graph=PTR, nodes=1 << 21), **kw)
    L = _C.lib()
    at = (C.c_int64 * (8 + 8 * a["hops"]))(*range(8 + 8 * a["hops"]))
    got = L.sgl_query_at(a["graph"], PTR, PTR, PTR, None, a["nodes"], PTR, PTR, PTR, 0, 1000, 0, 10, None, None, 0, None, None, 0, a["fanout"],
                         a["hops"], a["policy"], 0, -1, 0, 20, 24, 0, PTR, PTR, 1, 1, PTR, at, PTR, PTR, PTR, PTR, 1 << 62, None, None)
    assert got == rc, L.sgl_last_error()
    assert text in L.sgl_last_error().decode()
