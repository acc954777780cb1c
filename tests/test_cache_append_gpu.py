"""Appending a chunk of rows to caches of different lengths: the kernel against tensor indexing, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    return m


def _case(gen, b, s, hkv, d, rows, layout, strided):
    shape = (b, s, hkv, d) if layout == "bshd" else (b, hkv, s, d)
    kc, vc = (torch.randn(shape, generator=gen).half().cuda() for _ in range(2))
    if layout == "bhsd":
        kc, vc = kc.transpose(1, 2), vc.transpose(1, 2)
    if strided:   # k and v as halves of one projection's output
        kv = torch.randn(b, rows, 2 * hkv, d, generator=gen).half().cuda()
        return kc, vc, kv[:, :, :hkv], kv[:, :, hkv:]
    return kc, vc, *(torch.randn(b, rows, hkv, d, generator=gen).half().cuda() for _ in range(2))


@pytest.mark.parametrize("layout", ["bshd", "bhsd"])
@pytest.mark.parametrize("hkv,d,rows", [(1, 32, 2), (3, 96, 37), (8, 128, 256), (2, 256, 1), (5, 64, 129)])
def test_rows_land_where_indexing_puts_them(ext, layout, hkv, d, rows):
    gen = torch.Generator().manual_seed(rows + d)
    lens = torch.tensor([0, 5, 300 - rows, -rows], dtype=torch.int32).cuda()   # (negative: counted from the end)
    for strided in (False, True):
        kc, vc, k, v = _case(gen, 4, 300, hkv, d, rows, layout, strided)
        want = []
        pos = lens.long()[:, None] + torch.arange(rows, device="cuda")[None]
        for c, x in ((kc, k), (vc, v)):
            c = c.clone()
            c[torch.arange(4, device="cuda")[:, None], pos] = x
            want.append(c)
        new, fits = ext.cache_append(k, v, kc, vc, lens)
        assert torch.equal(kc, want[0]) and torch.equal(vc, want[1])
        assert torch.equal(new, lens + rows) and bool(fits)


def test_an_entry_without_room_is_reported_and_nothing_written_outside(ext):
    gen = torch.Generator().manual_seed(3)
    kc, vc, k, v = _case(gen, 3, 64, 2, 64, 8, "bshd", False)
    for bad, place in ((57, 7), (64, 0), (1 << 30, 0)):   # how many rows of the middle entry still have a place
        k2, v2 = kc.clone(), vc.clone()
        _, fits = ext.cache_append(k, v, k2, v2, torch.tensor([3, bad, 50], dtype=torch.int32).cuda())
        assert not bool(fits)
        assert torch.equal(k2[1, 64 - place:], k[1, :place]) and torch.equal(k2[1, :64 - place], kc[1, :64 - place])
        assert torch.equal(v2[0, 3:11], v[0]) and torch.equal(v2[2, 50:58], v[2])


def test_tensors_the_kernel_cannot_address_are_left_to_indexing(ext):
    gen = torch.Generator().manual_seed(4)
    kc, vc, k, v = _case(gen, 2, 64, 4, 64, 8, "bshd", False)
    lens = torch.zeros(2, dtype=torch.int32).cuda()
    before = kc.clone()
    for bad in ((k[:, :, :1], v[:, :, :1], kc, vc), (k.float(), v, kc, vc), (k, v, kc.transpose(2, 3), vc),
                (kc[:, :8], v, kc, vc), (k, v, kc[..., :60], vc[..., :60]), (k[..., 1:61], v[..., 1:61], kc, vc)):
        assert ext.cache_append(*bad, lens) is None
    assert ext.cache_append(k, v, kc, vc, lens.long()) is None
    assert torch.equal(kc, before)


def test_one_tensor_for_both_caches_ends_up_with_the_values(ext):
    gen = torch.Generator().manual_seed(5)
    kc, _, k, v = _case(gen, 2, 64, 4, 64, 8, "bshd", False)
    lens = torch.tensor([0, 30], dtype=torch.int32).cuda()
    assert ext.cache_append(k, v, kc, kc, lens) is None       # (the kernel writes both at once)
    kv = torch.zeros(2, 64, 2, 4, 64, dtype=torch.float16, device="cuda")   # K and V of a position side by side
    assert ext.cache_append(k, v, kv[:, :, 0], kv[:, :, 1], lens) is not None
    assert torch.equal(kv[1, 30:38, 0], k[1]) and torch.equal(kv[1, 30:38, 1], v[1])
