"""The two-kernel sort of mini-batch sized lists at the edges of its forms: one CTA (up to 2,048 items), 256-item tiles, the
largest list, and key widths with which key and position share a word or do not."""
import numpy as np
import pytest
import torch

from gpu_util import cu, npy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 767, 768, 2048, 2049, 148 * 256, 148 * 256 + 1, 160001, 606208, 606209, 1212416, 1212417])
@pytest.mark.parametrize("bits", [1, 44, 64])
@pytest.mark.parametrize("pattern", ["random", "few values", "ascending", "descending"])
def test_stable_at_every_form(n, bits, pattern):
    from starrygl import ops
    gen = torch.Generator(device="cuda").manual_seed(n + bits)
    k = torch.randint(0, 1 << min(bits, 62), (n,), device="cuda", generator=gen)
    if bits == 64:
        k = k * 4 - 5                                   # the full range of bit patterns
    if pattern == "few values":
        k = k % 7
    elif pattern != "random":
        k = k.sort(descending=pattern == "descending").values
    v = torch.randint(0, 1 << 31, (n,), device="cuda", dtype=torch.int64, generator=gen).int()
    ks, vs = ops.radix_sort_pairs(k, v, bits)
    order = torch.sort(k if bits < 64 else k ^ (-1 << 63), stable=True).indices
    assert torch.equal(ks, k[order]) and torch.equal(vs, v[order])


@pytest.mark.parametrize("n", [2049, 5000, 60000])
def test_equal_keys_of_all_ones_across_buckets(n):
    """64-bit keys whose largest value, all ones, fills several buckets."""
    from starrygl import ops
    top = 2 ** 63 - 1
    rng = np.random.default_rng(n)
    ids = np.where(rng.random(n) < 0.9, 1, rng.integers(0, 2, n)).astype(np.int64)
    ts = np.where(rng.random(n) < 0.95, top, rng.integers(0, 2, n) * top).astype(np.int64)
    st = ops.StatusWord(torch.device("cuda"))
    out_id, out_ts, inv, _, d_n = ops.unique_pairs(cu(ids), cu(ts), id_bits=1, ts_bits=63, ts_base=0, status=st)[:5]
    uniq, want = np.unique(np.stack([ids, ts], 1), axis=0, return_inverse=True)
    assert int(d_n) == len(uniq) and np.array_equal(npy(inv[:n]), want.reshape(-1))
    assert np.array_equal(npy(out_id[:len(uniq)]), uniq[:, 0]) and np.array_equal(npy(out_ts[:len(uniq)]), uniq[:, 1])
    st.check("unique_pairs")
    g = ops.tcsr_build(cu(ids), cu(np.arange(n, dtype=np.int64)), cu(ts), None, 2)
    order = np.lexsort((ts, ids))
    assert np.array_equal(npy(g.indptr), np.searchsorted(ids[order], [0, 1, 2])) and np.array_equal(npy(g.nbr), order)


@pytest.mark.parametrize("n", [600, 2048, 2049, 41000, 300000, 610000])
@pytest.mark.parametrize("copies", [1, 30])
def test_pairs_of_a_power_law(n, copies):
    """A few ids hold a large part of the list, all within a short time: bins are cut again, or given up for pivots."""
    from starrygl import ops
    rng = np.random.default_rng(n + copies)
    m = max(n // copies, 1)
    pick = rng.integers(0, m, n) if copies > 1 else np.arange(n)
    ids = np.minimum((rng.random(m) + 1e-9) ** -1.1, 799999).astype(np.int64)[pick]
    ts = rng.integers(5_000_000, 5_000_000 + max(m // 50, 3), m).astype(np.int64)[pick]
    cut = n // 3
    st = ops.StatusWord(torch.device("cuda"))
    out_id, out_ts, inv_a, inv_b, d_n = ops.unique_pairs(cu(ids[:cut]), cu(ts[:cut]), cu(ids[cut:]), cu(ts[cut:]), id_bits=20, ts_bits=24,
                                                         ts_base=0, status=st)[:5]
    uniq, inv = np.unique((ids << 24) | ts, return_inverse=True)
    assert int(d_n) == len(uniq)
    assert np.array_equal(npy(out_id[:len(uniq)]), uniq >> 24) and np.array_equal(npy(out_ts[:len(uniq)]), uniq & (2 ** 24 - 1))
    assert np.array_equal(npy(inv_a[:cut]), inv[:cut]) and np.array_equal(npy(inv_b[:n - cut]), inv[cut:])
    st.check("unique_pairs")


@pytest.mark.parametrize("n", [64, 65, 511, 512, 513, 1537, 2048])
@pytest.mark.parametrize("ts_bits", [24, 40])
@pytest.mark.parametrize("share", [0, 0.05, 0.1, 0.6, 1])
def test_one_cta_with_items_close_to_each_other(n, ts_bits, share):
    """A list of one CTA by counting and by pivots, on both sides of the share of one id at which it changes; keys of one word and of two."""
    from starrygl import ops
    rng = np.random.default_rng(n)
    ids = np.where(rng.random(n) < share, 777, rng.integers(0, 800000, n)).astype(np.int64)
    ts = rng.integers(0, 2 ** ts_bits if n % 2 else 50, n).astype(np.int64)
    st = ops.StatusWord(torch.device("cuda"))
    out_id, out_ts, inv, _, d_n = ops.unique_pairs(cu(ids), cu(ts), None, None, id_bits=20, ts_bits=ts_bits, ts_base=0, status=st)[:5]
    uniq, want = np.unique((ids << ts_bits) | ts, return_inverse=True)
    assert int(d_n) == len(uniq) and np.array_equal(npy(inv[:n]), want)
    assert np.array_equal(npy(out_id[:len(uniq)]), uniq >> ts_bits) and np.array_equal(npy(out_ts[:len(uniq)]), uniq & (2 ** ts_bits - 1))
    st.check("unique_pairs")
