"""Decode on batches too small to fill the GPU: the splits get finer and the combine step merges many of them."""
import math

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    return m


# Lengths on both sides of 256- and 512-position splits, the empty and the full cache; one KV head of 16 and 20
# query heads (one and two MMA row blocks); the head dims with kernels of their own and one that borrows.
@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (16, 1, 64), (20, 1, 96), (4, 2, 256), (8, 8, 32)])
@pytest.mark.parametrize("lens,capacity", [([1999], 4096), ([255, 256, 257], 700), ([0, 1, 511, 2049], 2049),
                                           ([9000], 9001)])
def test_small_batches_against_the_oracle(ext, hq, hkv, d, lens, capacity):
    gen = torch.Generator().manual_seed(hq * d + capacity)
    b, scale = len(lens), 1 / math.sqrt(d)
    q = torch.randn(b, hq, d, generator=gen).half()
    kc, vc = (torch.randn(b, capacity, hkv, d, generator=gen).half() for _ in range(2))
    for i, n in enumerate(lens):   # what lies behind a length does not matter
        kc[i, n:] = float("nan")
        vc[i, n:] = float("inf")
    lens = torch.tensor(lens, dtype=torch.int32)
    args = q.cuda(), kc.cuda(), vc.cuda(), lens.cuda(), scale
    o, lse = ext.decode(*args, return_lse=True)
    o_ref, lse_ref = orc.decode_fwd(q, kc, vc, lens, scale)
    assert orc.rel_max_err(o, o_ref) <= orc.TOL_O
    seen = lens > 0
    assert orc.abs_max_err(lse[seen.cuda()], lse_ref[seen]) <= orc.TOL_LSE
    assert torch.isneginf(lse[~seen.cuda()]).all() and not o[~seen.cuda()].any()
    # the fixed scratch is larger than the workspace of the call above; the splits are the same
    out = torch.empty_like(o)
    assert torch.equal(ext.decode_static(*args, out=out), o)
    assert ext.device_status() == 0


# Entries on both sides of where a cut gets coarser, in one call (batch x KV heads leave 3 to 30 splits per entry to
# the SMs); the new token in the last position of a split and in the first of the next; one warp and one block per row
# of the merge, and a number of rows that is not a multiple of four.
@pytest.mark.parametrize("hq,hkv,d", [(8, 8, 128), (6, 2, 64), (9, 3, 256), (4, 1, 32), (32, 8, 96)])
@pytest.mark.parametrize("append", [False, True])
@pytest.mark.parametrize("capacity", [9216, 2500])
def test_cuts_of_different_fineness_in_one_batch(ext, hq, hkv, d, append, capacity):
    gen = torch.Generator().manual_seed(hq * d)
    lens = [n for n in (0, 1, 255, 256, 767, 768, 769, 1024, 1535, 1536, 1537, 2304, 3072, 3073, 4607, 4608, 6143, 6145, 9215)
            if n < capacity]
    b, scale = len(lens), 1 / math.sqrt(d)
    q = torch.randn(b, hq, d, generator=gen).half()
    kc, vc = (torch.randn(b, capacity, hkv, d, generator=gen).half() for _ in range(2))
    kn, vn = (torch.randn(b, hkv, d, generator=gen).half() for _ in range(2)) if append else (None, None)
    lens = torch.tensor(lens, dtype=torch.int32)
    dev = [t.cuda() if t is not None else None for t in (q, kc, vc, lens, kn, vn)]
    o, lse = ext.decode(*dev[:4], scale, k_new=dev[4], v_new=dev[5], return_lse=True)
    if append:
        for i, n in enumerate(lens.tolist()):
            kc[i, n], vc[i, n] = kn[i], vn[i]
        assert torch.equal(dev[1].cpu(), kc) and torch.equal(dev[2].cpu(), vc)
        lens = lens + 1
    o_ref, lse_ref = orc.decode_fwd(q, kc, vc, lens, scale)
    assert orc.rel_max_err(o, o_ref) <= orc.TOL_O
    seen = lens > 0
    assert orc.abs_max_err(lse.cpu()[seen], lse_ref[seen]) <= orc.TOL_LSE
    assert ext.device_status() == 0
