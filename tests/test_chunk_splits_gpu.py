"""A chunk of new tokens too small to fill the GPU: several thread blocks share each query block's keys."""
import math

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    return m


# One and two query blocks; entries whose keys end inside the first split, at a tile's edge, in the last split; an
# entry shorter than the chunk (its first queries see no key) and an empty one; every head_dim; up to 32 splits.
@pytest.mark.parametrize("hq,hkv,d,nq,lens,capacity", [
    (4, 1, 128, 2, [1999], 2100), (8, 2, 64, 130, [130, 512, 3000], 3001), (2, 2, 256, 128, [640, 100], 700),
    (6, 3, 96, 37, [5, 0, 1300, 129], 1300), (1, 1, 32, 300, [9000], 9001)])
@pytest.mark.parametrize("causal", [True, False])
def test_split_chunk_against_the_oracle(ext, hq, hkv, d, nq, lens, capacity, causal):
    gen = torch.Generator().manual_seed(d + nq)
    b, scale = len(lens), 1 / math.sqrt(d)
    assert ext._lib.fal_fwd_kvcache_workspace_bytes(b, hq, nq, capacity, d) > 0
    q = torch.randn(b, hq, nq, d, generator=gen).half()
    kc, vc = (torch.randn(b, hkv, capacity, d, generator=gen).half() for _ in range(2))
    for i, n in enumerate(lens):   # what lies behind a length does not matter
        kc[i, :, n:] = float("nan")
        vc[i, :, n:] = float("inf")
    lens = torch.tensor(lens, dtype=torch.int32)
    wide = torch.full((b, hq, nq, d + 8), 7.0, dtype=torch.float16, device="cuda")   # guard columns
    o, lse = ext.forward_kvcache(q.cuda(), kc.cuda(), vc.cuda(), lens.cuda(), scale, causal, out=wide[..., :d])
    o_ref, lse_ref = orc.kvcache_chunk_fwd(q, kc, vc, lens, scale, causal)
    assert orc.rel_max_err(o, o_ref) <= orc.TOL_O
    seen = torch.isfinite(lse_ref)
    assert orc.abs_max_err(lse.cpu()[seen], lse_ref[seen]) <= orc.TOL_LSE
    assert torch.isneginf(lse.cpu()[~seen]).all() and not o.cpu()[~seen].any()
    assert (wide[..., d:] == 7.0).all()
    assert ext.device_status() == 0


def _call(ext, q, kc, vc, lens, mask, workspace=None):
    """fal_fwd_kvcache, or the split call with a workspace; returns (O, LSE)."""
    (b, hq, nq, d), (hkv, capacity) = q.shape, kc.shape[1:3]
    o, lse = torch.full_like(q, 5.0), torch.full((b, hq, nq), 5.0, device="cuda")
    args = ext._FWD_ARGS.pack(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), o.data_ptr(), lse.data_ptr(), lens.data_ptr(),
                              b, hq, hkv, nq, capacity, d, *q.stride()[:3], *kc.stride()[:3], *vc.stride()[:3],
                              *o.stride()[:3], 1 / math.sqrt(d), mask, ext._status_ptr(0), ext._raw_stream(0))
    if workspace is None:
        ext._check(ext._fwd_run(args))
    else:
        ext._check(ext._lib.fal_fwd_kvcache_split_run(args, workspace.data_ptr(), workspace.numel() * 4))
    assert ext.device_status() == 0
    return o.cpu(), lse.cpu()


def _inputs(ext, hq, hkv, d, nq, lens, capacity):
    """Inputs of a chunk that is split, and a workspace full of NaN."""
    gen = torch.Generator().manual_seed(d + nq)
    b = len(lens)
    q = torch.randn(b, hq, nq, d, generator=gen).half().cuda()
    kc, vc = (torch.randn(b, hkv, capacity, d, generator=gen).half().cuda() for _ in range(2))
    nbytes = ext._lib.fal_fwd_kvcache_workspace_bytes(b, hq, nq, capacity, d)
    assert nbytes > 0
    return q, kc, vc, torch.tensor(lens, dtype=torch.int32).cuda(), torch.full((nbytes // 4,), math.nan, device="cuda")


@pytest.mark.parametrize("mask", [0, 1, 2])
@pytest.mark.parametrize("d", [64, 96, 128, 256])
def test_the_split_call_takes_every_mask(ext, mask, d):
    q, kc, vc, lens, ws = _inputs(ext, 4, 2, d, 200, [1500, 333], 1500)
    o, lse = _call(ext, q, kc, vc, lens, mask, ws)
    o_whole, lse_whole = _call(ext, q, kc, vc, lens, mask)
    assert orc.rel_max_err(o, o_whole) <= orc.TOL_O
    assert orc.abs_max_err(lse, lse_whole) <= orc.TOL_LSE


@pytest.mark.parametrize("where,value", [("v", math.inf), ("v", math.nan), ("k", math.inf), ("k", math.nan)])
@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("hq,nq,keys,at", [(8, 512, 600, 300), (8, 512, 600, 599), (2, 130, 3000, 2990), (4, 300, 200, 150)])
def test_what_a_row_cannot_see_does_not_reach_it(ext, where, value, d, hq, nq, keys, at):
    """An infinity or NaN in one key or value row: in the split chunk it reaches every row that sees the key and no
    row that it does not reach in the unsplit one (whose blocks read whole key tiles)."""
    q, kc, vc, lens, ws = _inputs(ext, hq, hq, d, nq, [keys], 700 if keys < 700 else keys)
    (kc if where == "k" else vc)[0, :, at] = value
    o, lse = _call(ext, q, kc, vc, lens, 2, ws)
    o_whole, lse_whole = _call(ext, q, kc, vc, lens, 2)
    sees = torch.arange(nq) + keys - nq >= at
    reached, reached_whole = ~torch.isfinite(o).all(-1), ~torch.isfinite(o_whole).all(-1)
    assert torch.equal(reached[..., sees], reached_whole[..., sees]) and not (reached & ~reached_whole).any()
    clean = ~reached_whole
    seen = clean & torch.isfinite(lse_whole)
    if seen.any():
        assert orc.rel_max_err(o[clean], o_whole[clean]) <= orc.TOL_O
        assert orc.abs_max_err(lse[seen], lse_whole[seen]) <= orc.TOL_LSE
    if where == "v":   # scores and their sums are as without it
        assert torch.equal(torch.isfinite(lse), torch.isfinite(lse_whole))


@pytest.mark.parametrize("variant", ["FWD_ONE_TILE", "FWD_TWO_TILES", "FWD_HALF_SM"])
def test_a_forced_variant_is_not_split(ext, variant):
    q, kc, vc, lens, ws = _inputs(ext, 4, 2, 64, 200, [1500, 333], 1500)
    ext.set_forward_variant(getattr(ext, variant))
    try:
        o, lse = _call(ext, q, kc, vc, lens, 2, ws)
        o_whole, lse_whole = _call(ext, q, kc, vc, lens, 2)
    finally:
        ext.set_forward_variant(ext.FWD_AUTO)
    assert torch.equal(o, o_whole) and torch.equal(lse, lse_whole)
    assert torch.isnan(ws).all()   # nobody wrote a partial result


@pytest.mark.parametrize("nq,hq,capacity,splits,most", [(16, 32, 3000, 4, 512), (130, 32, 3000, 2, 896), (40, 8, 9000, 18, 512)])
@pytest.mark.parametrize("mask", [0, 2])
def test_entries_of_few_keys_are_not_shared(ext, nq, hq, capacity, splits, most, mask):
    """A large cache that holds little so far: one thread block finishes each query block without partial results,
    up to `most` keys; with one more the keys are shared.  (The first 4 KB of the workspace hold the first rows of
    split 0, which computes the keys that every row sees.)"""
    for keys in (most + 1, most, nq, 1):
        q, kc, vc, lens, ws = _inputs(ext, hq, hq, 64, nq, [keys], capacity)
        assert ws.numel() == splits * hq * nq * 65
        o, lse = _call(ext, q, kc, vc, lens, mask, ws)
        assert torch.isnan(ws).all().item() == (keys <= most) and torch.isnan(ws[:1024]).any().item() == (keys <= most)
        o_whole, lse_whole = _call(ext, q, kc, vc, lens, mask)
        assert orc.rel_max_err(o, o_whole) <= orc.TOL_O
        seen = torch.isfinite(lse_whole)
        assert torch.equal(seen, torch.isfinite(lse)) and orc.abs_max_err(lse[seen], lse_whole[seen]) <= orc.TOL_LSE
