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


# One, two and four entries on a lane, the last of them alone, and one entry more than are put in order; lengths
# that differ by less and by more than a block; one block per entry.
@pytest.mark.parametrize("b,h,nq,lens", [(128, 4, 130, (130, 900)), (129, 4, 130, (130, 900)), (97, 4, 200, (200, 210)),
                                         (33, 10, 5, (0, 900)), (2, 80, 300, (10, 900))])
@pytest.mark.parametrize("d", [64, 128])
def test_more_blocks_than_the_sms_take_at_once(ext, b, h, nq, lens, d):
    gen = torch.Generator().manual_seed(b + d)
    used = torch.randint(lens[0], lens[1] + 1, (b,), generator=gen, dtype=torch.int32)
    used[0], used[-1] = lens[1], lens[0]
    q = torch.randn(b, h, nq, d, generator=gen).half()
    kc, vc = (torch.randn(b, 1, 900, d, generator=gen).half() for _ in range(2))
    out = torch.full((b, h, nq, d), 9.0, dtype=torch.float16, device="cuda")
    ext.forward_kvcache(q.cuda(), kc.cuda(), vc.cuda(), used.cuda(), 1 / math.sqrt(d), out=out)
    ref, _ = orc.kvcache_chunk_fwd(q, kc, vc, used, 1 / math.sqrt(d))
    assert orc.rel_max_err(out, ref) <= orc.TOL_O
    assert ext.device_status() == 0


def test_the_order_of_many_entries_costs_little(ext):
    """Every thread block searches the lengths for its own: with 4 096 of them that took six times as long as the
    attention itself.  The unmasked call of the same size runs in the order of the entries."""
    q = torch.randn(4096, 8, 4, 64, device="cuda", dtype=torch.float16)
    kc, vc = (torch.randn(4096, 1, 128, 64, device="cuda", dtype=torch.float16) for _ in range(2))
    used = torch.randint(20, 121, (4096,), dtype=torch.int32, device="cuda")
    times = {True: [], False: []}
    for _ in range(6):
        for causal, seen in times.items():
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(5):
                ext.forward_kvcache(q, kc, vc, used, 0.125, causal)
            end.record()
            end.synchronize()
            seen.append(start.elapsed_time(end))
    assert min(times[True]) < 2 * min(times[False])
