"""What the extension module does with its arguments before it reaches for a device (the tensors are refused there: there is no CPU path)."""
import numpy as np
import pytest
import torch

from starrygl import _C, ops

E = torch.tensor([0, 1, 2])
ANY_TRUTH = [None, True, False, np.bool_(True), np.bool_(False), 0, 2, 0.0, 1.5, "", "x", [], (1,)]


@pytest.mark.parametrize("v", ANY_TRUTH, ids=repr)
def test_switches_are_any_truth_value(v):
    g = ops.TCSR(3, E, E, E, E, None, 0, 2, None)
    f = torch.zeros(3, 4)
    for call in (lambda: ops.tcsr_build(E, E, E, E, 3, want_perm=v), lambda: ops.tcsr_build(E, E, E, E, 3, want_fence=v),
                 lambda: _C.host().sample_layer(g.indptr, g.nbr, g.ts, g.eid, None, 3, E, E, 2, 0, None, 0, -1, 0, 0, 0, v, None, None, 0),
                 lambda: ops.mail_reduce(E, None, E, 3, [(f, None)], want_pos=v),
                 lambda: ops.mailbox_write(E, f, torch.zeros(3), torch.zeros(3, 1, 4), torch.zeros(3, 1), None, advance=v)):
        with pytest.raises(_C.SglError, match="expected a CUDA"):
            call()


def test_sizes_beyond_64_bits_are_refused():
    for nodes in (2 ** 64 + 4, 2 ** 63, 2 ** 63 - 1, -2 ** 63 - 1):
        with pytest.raises((OverflowError, RuntimeError)) as e:
            ops.tcsr_build(E, E, E, E, nodes)
        assert "expected a CUDA" not in str(e.value)
    for fanout in (2 ** 62, 2 ** 64 + 1, -2 ** 63):
        with pytest.raises((OverflowError, _C.SglError)) as e:
            _C.host().sample_layer(E, E, E, E, None, 3, E, E, fanout, 0, None, 0, -1, 0, 0, 0, False, None, None, 0)
        assert "expected a CUDA" not in str(e.value)


def test_seeds_and_addresses_are_taken_modulo_2_64():
    for seed in (-1, 2 ** 64 + 5, 2 ** 200):
        with pytest.raises(_C.SglError, match="expected a CUDA"):
            _C.host().sample_layer(E, E, E, E, None, 3, E, E, 2, 0, None, 0, -1, 0, seed, 0, False, None, None, 0)


@pytest.mark.parametrize("call,text", [
    (lambda: ops.tcsr_build(E, E[:2], E, None, 3), "differ in length"),
    (lambda: ops.tcsr_build(E.int(), E, E, None, 3), "expected int64 tensor, got torch.int32"),
    (lambda: ops.gather_rows(torch.zeros(3, 4).t(), E), "rows must be contiguous"),
    (lambda: ops.gather_rows(torch.zeros(3, 4), E.float()), "expected int64 tensor, got torch.float32"),
    (lambda: ops.cache_gather(torch.zeros(3, 4), E, None, E), "hitmap must be int32"),
    (lambda: ops.cache_gather(torch.zeros(3, 4), E.int(), torch.zeros(3, 5), E), "dense and of equal size"),
    (lambda: ops.mail_reduce(E, None, E.double(), 3), "timestamps must be int64 or float32"),
    (lambda: ops.mail_reduce(E, None, E, 3, [(torch.zeros(2, 4), None)]), "fewer rows than its entry list"),
    (lambda: ops.mail_reduce(E, E, E, 3, [(torch.zeros(3, 4), torch.zeros(3, 5))]), "equal width"),
    (lambda: ops.mailbox_write(E, torch.zeros(3, 4), torch.zeros(3), torch.zeros(3, 4), torch.zeros(3, 1), None), "contiguous"),
    (lambda: ops.mailbox_write(E, torch.zeros(3, 5), torch.zeros(3), torch.zeros(3, 1, 4), torch.zeros(3, 1), None), "mailbox's width"),
])
def test_refusals(call, text):
    with pytest.raises(_C.SglError, match=text):
        call()
