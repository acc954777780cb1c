"""Backward: dQ leaves in pieces of 32 rows (head_dim 96 and 128); query lengths on both sides of their edges, batched
and packed next to sequences whose rows must stay untouched."""
import math

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    return m


def _check(got, ref):
    # the scale of a gradient that a short sequence makes tiny is one score's rounding
    for g, r in zip(got, ref):
        assert (g.float().cpu() - r).abs().max().item() <= orc.TOL_GRAD * max(r.abs().max().item(), 0.5)


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 96, 97, 127, 161, 225])
def test_batched(ext, d, n):
    gen = torch.Generator().manual_seed(n + d)
    q, do = (torch.randn(2, 4, n, d, generator=gen).half() for _ in range(2))
    k, v = (torch.randn(2, 2, n, d, generator=gen).half() for _ in range(2))
    scale = 1 / math.sqrt(d)
    for causal in (False, True):
        o, lse = ext.forward(q.cuda(), k.cuda(), v.cuda(), scale, causal)
        got = ext.backward(do.cuda(), q.cuda(), k.cuda(), v.cuda(), o, lse, scale, causal)
        _check(got, orc.attention_bwd(q, k, v, do, scale, causal))
    assert ext.device_status() == 0


@pytest.mark.parametrize("d", [64, 128, 256])
def test_packed(ext, d):
    lens = [1, 33, 0, 127, 32, 160, 95, 129]
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0, dtype=torch.int32)
    total, scale = int(cu[-1]), 1 / math.sqrt(d)
    gen = torch.Generator().manual_seed(d)
    q, k, v, do = (torch.randn(total, 2, d, generator=gen).half() for _ in range(4))
    for causal in (False, True):
        a = q.cuda(), k.cuda(), v.cuda()
        o, lse = ext.forward_varlen(*a, cu.cuda(), cu.cuda(), max(lens), max(lens), scale, causal)
        got = ext.backward_varlen(do.cuda(), *a, o, lse, cu.cuda(), cu.cuda(), max(lens), max(lens), scale, causal)
        _check(got, orc.varlen_bwd(q, k, v, do, cu, cu, scale, causal))
    assert ext.device_status() == 0
