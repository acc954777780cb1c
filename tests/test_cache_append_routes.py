"""Which chunks of new tokens may be written by the append kernel, and which autograd has a say in."""
import pytest
import torch

import flash_attn_legacy_cuda as ext
from flash_attn_legacy import flash_attn_with_kvcache


@pytest.fixture()
def appended(monkeypatch):
    """Stands in for the append kernel and lists its calls (the attention behind it then refuses CPU tensors)."""
    calls = []

    def fake(k, v, k_cache, v_cache, lens):
        calls.append((k, v))
        return lens + k.shape[1], torch.ones(1, dtype=torch.bool)

    monkeypatch.setattr(ext, "cache_append", fake)
    return calls


def _tensors():
    gen = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(2, 3, 4, 64, generator=gen).half() for _ in range(3))
    kc, vc = (torch.zeros(2, 16, 4, 64, dtype=torch.float16) for _ in range(2))
    return q, kc, vc, k, v, torch.tensor([2, 5], dtype=torch.int32)


@pytest.mark.parametrize("which", [0, 1])
def test_a_cache_made_in_inference_mode_is_not_written_outside_of_it(appended, which):
    q, kc, vc, k, v, lens = _tensors()
    caches = [kc, vc]
    with torch.inference_mode():
        caches[which] = caches[which].clone()
    with pytest.raises(RuntimeError, match="[Ii]nference"):
        flash_attn_with_kvcache(q, *caches, k=k, v=v, cache_seqlens=lens)
    assert not appended
    with torch.inference_mode(), pytest.raises(RuntimeError, match="CUDA"):
        flash_attn_with_kvcache(q, *caches, k=k, v=v, cache_seqlens=lens)
    assert len(appended) == 1


def test_forward_mode_tangents_go_into_the_caches(appended):
    from torch.autograd import forward_ad
    q, kc, vc, k, v, lens = _tensors()
    with forward_ad.dual_level():
        tangent = torch.ones_like(v)
        with pytest.raises(RuntimeError, match="CUDA"):
            flash_attn_with_kvcache(q, kc, vc, k=k, v=forward_ad.make_dual(v, tangent), cache_seqlens=lens)
        assert not appended
        got = forward_ad.unpack_dual(vc).tangent
        assert got is not None and torch.equal(got[1, 5:8], tangent[1]) and not got[1, :5].any()


@pytest.mark.parametrize("make,apart", [
    (lambda t: (t[0], t[1]), True),                                          # halves of one allocation
    (lambda t: (t.view(2, 10, 2, 3, 32)[:, :, 0], t.view(2, 10, 2, 3, 32)[:, :, 1]), True),   # K and V of a position side by side
    (lambda t: (t.view(2, 10, 3, 64)[..., :32], t.view(2, 10, 3, 64)[..., 32:]), True),       # of a head
    (lambda t: (t.clone()[0], t[0]), True),
    (lambda t: (t[0], t[0]), False),                                         # one tensor for both
    (lambda t: (t[0, :, :9], t[0, :, 1:]), False),
    (lambda t: (t[0, 0], t[1, 0]), True),
    (lambda t: (t[0, 0], t[0].transpose(1, 2)[1].transpose(0, 1)), True),    # other strides, behind the first
    (lambda t: (t.flatten()[:960].view(1, 10, 3, 32), t.flatten()[512:1472].view(1, 10, 3, 32)), False),
])
def test_caches_that_share_rows_are_told_from_those_that_share_an_allocation(make, apart):
    k_cache, v_cache = make(torch.zeros(2, 2, 10, 3, 32, dtype=torch.float16))
    assert ext._rows_apart(k_cache, v_cache) is apart and ext._rows_apart(v_cache, k_cache) is apart
