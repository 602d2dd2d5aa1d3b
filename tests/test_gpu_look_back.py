"""Look-backs that run into their limit while they wait (a limit of 0 gives up without waiting and covers only how that is reported): with
a limit of a nanosecond some sort soon has to wait longer, and every one that need not is right."""
import pytest
import torch

from starrygl import _C, ops

pytestmark = pytest.mark.gpu


@pytest.fixture
def a_nanosecond():
    before = _C.lib().sgl_look_back_limit(1)
    yield
    _C.lib().sgl_look_back_limit(before)


def until_one_gives_up(call, rounds=60):
    for _ in range(rounds):
        try:
            call()
        except _C.SglError as e:
            assert "time limit" in str(e) or "timed out" in str(e)
            return True
    return False


def test_sort(a_nanosecond):
    n = 8_000_000
    keys = torch.randint(0, 2 ** 40, (n,), device="cuda")
    want, order = torch.sort(keys, stable=True)

    def call():
        k, v = ops.radix_sort_pairs(keys, torch.arange(n, dtype=torch.int32, device="cuda"), 40)
        assert torch.equal(k, want) and torch.equal(v.long(), order)
    assert until_one_gives_up(call)
    _C.lib().sgl_look_back_limit(2_000_000_000)
    call()


@pytest.mark.parametrize("perm", [False, True])
def test_build(a_nanosecond, perm):
    m, nodes = 4_000_000, 50_000
    gen = torch.Generator(device="cuda").manual_seed(3)
    key, nbr = (torch.randint(0, nodes, (m,), device="cuda", generator=gen) for _ in range(2))
    ts = torch.randint(0, 100_000, (m,), device="cuda", generator=gen)
    order = torch.argsort(key * 100_000 + ts, stable=True)

    def call():
        g = ops.tcsr_build(key, nbr, ts, None, nodes, want_perm=perm)
        assert torch.equal(g.eid, order) and torch.equal(g.nbr, nbr[order]) and torch.equal(g.ts, ts[order])
    assert until_one_gives_up(call)
    _C.lib().sgl_look_back_limit(2_000_000_000)
    call()


def test_list(a_nanosecond):
    n = 4_000_000
    ids = torch.randint(0, 1 << 21, (n,), device="cuda")
    zero = torch.zeros_like(ids)
    want, inv = torch.unique(ids, return_inverse=True)
    st = ops.StatusWord(ids.device)

    def call():
        out = ops.unique_pairs(ids, zero, id_bits=21, ts_bits=0, ts_base=0, status=st)
        st.check("lists")
        assert int(out[4]) == want.numel() and torch.equal(out[0][:want.numel()], want) and torch.equal(out[2][:n], inv)
    assert until_one_gives_up(call)
    _C.lib().sgl_look_back_limit(2_000_000_000)
    call()
