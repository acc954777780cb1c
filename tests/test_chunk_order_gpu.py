"""Chunks behind caches of many different lengths: every (entry, query block) is computed once, whatever the order
in which the blocks are handed out (heaviest first; entries on the lanes of a warp, 32 at a time)."""
import math

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    return m


@pytest.mark.parametrize("b,nq,lens", [(2, 700, (700, 900)), (33, 300, (300, 700)), (40, 260, (0, 600)), (70, 129, (129, 130))])
@pytest.mark.parametrize("d", [64, 128])
def test_every_block_of_every_entry(ext, b, nq, lens, d):
    gen = torch.Generator().manual_seed(b + d)
    cap, scale = 900, 1 / math.sqrt(d)
    used = torch.randint(lens[0], lens[1] + 1, (b,), generator=gen, dtype=torch.int32)
    q = torch.randn(b, 2, nq, d, generator=gen).half()
    kc, vc = (torch.randn(b, 1, cap, d, generator=gen).half() for _ in range(2))
    for variant in (ext.FWD_AUTO, ext.FWD_TWO_TILES):
        ext.set_forward_variant(variant)
        try:
            out = torch.full((b, 2, nq, d), 9.0, dtype=torch.float16, device="cuda")
            ext.forward_kvcache(q.cuda(), kc.cuda(), vc.cuda(), used.cuda(), scale, out=out)
        finally:
            ext.set_forward_variant(ext.FWD_AUTO)
        ref, _ = orc.kvcache_chunk_fwd(q, kc, vc, used, scale)
        assert orc.rel_max_err(out, ref) <= orc.TOL_O
    assert ext.device_status() == 0
