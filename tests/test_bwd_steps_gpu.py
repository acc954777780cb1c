"""Backward: thread blocks of few and many steps (query tiles x heads of a group), on both sides of the depths of the
operand rings, with partial query and key tiles under every mask."""
import math

import pytest
import torch

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    return m


@pytest.mark.parametrize("d", [32, 64, 128, 256])
@pytest.mark.parametrize("nq,group", [(5, 1), (129, 1), (300, 1), (512, 1), (64, 5), (200, 3), (641, 2)])
@pytest.mark.parametrize("mask", ["none", "causal", "end"])
def test_rectangular(ext, d, nq, group, mask):
    scale = 1 / math.sqrt(d)
    for nk in (100, 257) if mask != "end" else (nq, nq + 77):
        gen = torch.Generator().manual_seed(nq * 31 + nk + d)
        q, do = (torch.randn(1, 2 * group, nq, d, generator=gen).half() for _ in range(2))
        k, v = (torch.randn(1, 2, nk, d, generator=gen).half() for _ in range(2))
        end = mask == "end"
        a = q.cuda(), k.cuda(), v.cuda()
        o, lse = ext.forward_rect(*a, scale, mask != "none", bottom_right=end)
        got = ext.backward(do.cuda(), *a, o, lse, scale, mask != "none", bottom_right=end)
        ref = orc.attention_bwd(q, k, v, do, scale, mask != "none", nk - nq if end else 0)
        for g, r in zip(got, ref):  # P and dS are rounded to fp16 before their products, as TOL_GRAD allows for
            assert orc.rel_max_err(g, r) <= orc.TOL_GRAD
    assert ext.device_status() == 0
