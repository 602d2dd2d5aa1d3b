"""Kernels of a composite call submitted as one graph: more sequences than a thread keeps graphs for, threads side by side."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _pairs(n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, 5000, (n,), device="cuda", generator=gen), torch.randint(0, 16, (n,), device="cuda", generator=gen)


def _check(ids, ts):
    from starrygl import ops
    out_id, out_ts, inv, _, d_n = ops.unique_pairs(ids, ts, id_bits=13, ts_bits=4, ts_base=0)[:5]
    uniq, want = torch.unique((ids << 4) | ts, return_inverse=True)
    u = int(d_n)
    return u == uniq.numel() and torch.equal(out_id[:u], uniq >> 4) and torch.equal(out_ts[:u], uniq & 15) and torch.equal(inv[:ids.numel()], want)


def test_more_streams_than_graphs_are_kept():
    """20 streams with two sequences each in rotation, three rounds: graphs are made, launched with new sizes and dropped while others run."""
    from starrygl import _C
    streams = [torch.cuda.Stream() for _ in range(20)]
    for r in range(3):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                assert _check(*_pairs(3000 + 40 * i + r, i)) and _check(*_pairs(1_300_000 + 40 * i + r, i))     # two sequences each
        assert _C.lib().sgl_launch_graphs() <= 32
    with torch.cuda.stream(streams[0]):
        assert _check(*_pairs(5000, 1)) and _check(*_pairs(6000, 2)) and _check(*_pairs(40000, 3))


def test_threads_side_by_side():
    """Every thread has its graphs; calls of several threads, on one stream each and in turn on a common one, do not mix."""
    common, wrong = torch.cuda.Stream(), []

    def work(t):
        own = torch.cuda.Stream()
        for i in range(30):
            with torch.cuda.stream(own):
                if not _check(*_pairs(2049 + 100 * t + i, 100 * t + i)):
                    wrong.append((t, i))
    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong
    for t in range(3):                                  # a thread that ends gives its graphs back; the next starts anew
        done = []

        def once():
            with torch.cuda.stream(common):
                done.append([_check(*_pairs(3000 + t, i)) for i in range(4)])
        th = threading.Thread(target=once)
        th.start()
        th.join()
        assert done == [[True] * 4]


def test_a_thread_that_ends_gives_its_result_words_back():
    from starrygl import _C
    t = torch.arange(8, device="cuda")
    used, ok = set(), []

    def once():
        used.add(_C.host_words()[0])
        ok.append(_C.read_words(t, 8) == list(range(8)))
    for _ in range(64):
        th = threading.Thread(target=once)
        th.start()
        th.join()
    assert all(ok) and len(ok) == 64 and len(used) < 16        # the driver hands freed words out again
