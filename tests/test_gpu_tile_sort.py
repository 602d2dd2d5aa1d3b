"""The two-kernel sort of mini-batch sized lists at the edges of its forms: one CTA (up to 2,048 items), 256-item tiles, the
largest list, and key widths with which key and position share a word or do not."""
import pytest
import torch

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
