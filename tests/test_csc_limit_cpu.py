"""The CSC along a list keeps first edges in 32 bits: more edges than that are refused before anything is launched (so this needs no GPU).
The function is internal; its symbol is looked up by what it is called in the library."""
import ctypes as C
import subprocess

import pytest

from starrygl import _C


@pytest.fixture(scope="module")
def build_csc_rows():
    names = [l.split()[-1] for l in subprocess.run(["nm", "-D", "--defined-only", _C.LIB_PATH], capture_output=True, text=True).stdout.splitlines()]
    name, = [n for n in names if n.startswith("_ZN3sgl14build_csc_rowsE")]
    return getattr(C.CDLL(_C.LIB_PATH), name)


@pytest.mark.parametrize("edges,items", [(1 << 32, 1000), (1 << 40, 1000), (1000, 1 << 32), (-1, 1000)])
def test_refused(build_csc_rows, edges, items):
    order = (C.c_void_p * 3)(None, None, None)      # (by reference: a struct of three pointers)
    v, i64 = C.c_void_p, C.c_int64
    rc = build_csc_rows(C.byref(order), i64(items), v(), v(), 10, C.c_bool(False), v(), v(), v(), v(), v(), i64(edges), v(), i64(items), v(), 10, 10,
                        i64(0), v(), v(), v(), v(), v(), v(), v(), C.c_size_t(0), v())
    assert rc == -5 and b"64-bit positions" in _C.lib().sgl_last_error()
