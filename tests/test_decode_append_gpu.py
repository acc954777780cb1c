"""Decode with a new token: its row is streamed from where it came from and stored beside.  Positions on both sides of
slice (16 keys) and split edges, more than one chunk of query heads, left padding up to and behind the new position."""
import math

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    return m


@pytest.mark.parametrize("d", [32, 64, 96, 128, 256])
@pytest.mark.parametrize("layout", ["bshd", "bhsd"])
@pytest.mark.parametrize("hq,hkv", [(4, 4), (8, 2), (20, 1)])
def test_positions(ext, d, layout, hq, hkv):
    cap, lens = 600, torch.tensor([0, 1, 15, 16, 17, 63, 64, 255, 256, 257, 511, 512, 599], dtype=torch.int32)
    b, scale = len(lens), 1 / math.sqrt(d)
    gen = torch.Generator().manual_seed(d + hq)
    q, k, v = (torch.randn(b, h, d, generator=gen).half() for h in (hq, hkv, hkv))
    kc, vc = (torch.randn(b, cap, hkv, d, generator=gen).half() for _ in range(2))
    for i, n in enumerate(lens.tolist()):  # what stands where the new row goes must not be read
        kc[i, n] = float("nan")
        vc[i, n] = float("inf")
    for starts in (None, (lens // 2).int(), lens):
        a, c = (x.cuda() if layout == "bshd" else x.transpose(1, 2).contiguous().cuda() for x in (kc, vc))
        o = ext.decode(q.cuda(), a, c, lens.cuda(), scale, k.cuda(), v.cuda(), cache_layout=layout,
                       cache_starts=None if starts is None else starts.cuda())
        a, c = (x if layout == "bshd" else x.transpose(1, 2) for x in (a, c))
        for i, n in enumerate(lens.tolist()):
            assert torch.equal(a[i, n].cpu(), k[i]) and torch.equal(c[i, n].cpu(), v[i])
        ref = orc.decode_fwd(q, a.cpu(), c.cpu(), lens + 1, scale, starts)
        assert orc.rel_max_err(o, ref[0] if isinstance(ref, tuple) else ref) <= orc.TOL_O
    assert ext.device_status() == 0
