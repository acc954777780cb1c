"""The forward's half-SM CTAs (head_dim 32 and 64) at the edges of query and key tiles, against the oracle."""
import math

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    m.set_forward_variant(m.FWD_HALF_SM)
    yield m
    m.set_forward_variant(m.FWD_AUTO)


@pytest.mark.parametrize("d", [32, 64])
@pytest.mark.parametrize("nq,nk", [(1, 1), (127, 128), (128, 129), (129, 127), (257, 640), (300, 5)])
@pytest.mark.parametrize("mask", ["none", "causal", "end"])
def test_batched(ext, d, nq, nk, mask):
    if mask == "end" and nk < nq:
        pytest.skip("the end-aligned mask needs as many keys as queries")
    gen = torch.Generator().manual_seed(nq + nk)
    q, k, v = (torch.randn(2, h, n, d, generator=gen).half() for h, n in ((4, nq), (2, nk), (2, nk)))
    scale = 1 / math.sqrt(d)
    o, lse = ext.forward_rect(q.cuda(), k.cuda(), v.cuda(), scale, mask != "none", bottom_right=mask == "end")
    o_ref, lse_ref = orc.attention_fwd(q, k, v, scale, mask != "none", nk - nq if mask == "end" else 0)
    assert orc.rel_max_err(o, o_ref) <= orc.TOL_O
    assert orc.abs_max_err(lse, lse_ref) <= orc.TOL_LSE
    assert ext.device_status() == 0


@pytest.mark.parametrize("causal", [False, True])
def test_packed_and_ragged_caches(ext, causal):
    gen = torch.Generator().manual_seed(9)
    lens = [1, 128, 0, 300, 129]
    cu = torch.tensor([0, 1, 129, 129, 429, 558], dtype=torch.int32)
    q, k, v = (torch.randn(558, 4, 64, generator=gen).half() for _ in range(3))
    o, _ = ext.forward_varlen(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), 0.125, causal)
    assert orc.rel_max_err(o, orc.varlen_fwd(q, k, v, cu, cu, 0.125, causal)[0]) <= orc.TOL_O
    # caches holding NaN and infinity behind their lengths
    used = torch.tensor([130, 256, 511], dtype=torch.int32)
    q, kc, vc = (torch.randn(3, h, n, 64, generator=gen).half() for h, n in ((4, 130), (2, 512), (2, 512)))
    for b in range(3):
        kc[b, :, used[b]:] = float("nan")
        vc[b, :, used[b]:] = float("inf")
    o, _ = ext.forward_kvcache(q.cuda(), kc.cuda(), vc.cuda(), used.cuda(), 0.125)
    assert orc.rel_max_err(o, orc.kvcache_chunk_fwd(q, kc, vc, used, 0.125)[0]) <= orc.TOL_O
    assert ext.device_status() == 0
