"""Backward on long rows: thread blocks handed out two (batch, KV head) groups at a time, an odd group left over."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ext():
    import flash_attn_legacy_cuda as m
    return m


def _same(got, want):
    """dK and dV bit for bit (a block sums its queries in the same order); dQ is summed in any order."""
    (dq, dk, dv), (dq2, dk2, dv2) = got, want
    assert torch.equal(dk, dk2) and torch.equal(dv, dv2)
    # fp32 sums in another order, then one rounding to fp16: a unit in the last place of the largest value or so
    assert (dq.float() - dq2.float()).abs().max() <= 2 ** -10 * dq2.float().abs().max()


def test_five_groups_against_one_at_a_time(ext):
    n, d, scale = 104900, 128, 1 / math.sqrt(128)   # 5 x 4 heads: more than 2 GiB of Q, dO and dQ
    torch.manual_seed(0)
    q, do = (torch.randn(1, 20, n, d, device="cuda", dtype=torch.float16) for _ in range(2))
    k, v = (torch.randn(1, 5, n, d, device="cuda", dtype=torch.float16) for _ in range(2))
    o, lse = ext.forward(q, k, v, scale, True)
    got = ext.backward(do, q, k, v, o, lse, scale, True)
    for h in range(5):
        one = slice(4 * h, 4 * h + 4), slice(h, h + 1)
        want = ext.backward(do[:, one[0]], q[:, one[0]], k[:, one[1]], v[:, one[1]], o[:, one[0]],
                            lse[:, one[0]].contiguous(), scale, True)
        _same((got[0][:, one[0]], got[1][:, one[1]], got[2][:, one[1]]), want)
    assert ext.device_status() == 0


@pytest.mark.parametrize("causal", [True, False])
def test_packed_sequences_with_a_long_bound(ext, causal):
    """The caller's bound on the row count decides how the blocks are handed out, and nothing else."""
    torch.manual_seed(1)
    lens = torch.randint(0, 400, (290,))
    lens[3] = 0
    cu = torch.nn.functional.pad(lens.cumsum(0), (1, 0)).int().cuda()
    n = int(lens.sum())
    q, do = (torch.randn(n, 80, 64, device="cuda", dtype=torch.float16) for _ in range(2))
    k, v = (torch.randn(n, 5, 64, device="cuda", dtype=torch.float16) for _ in range(2))
    assert n * 80 * 64 * 8 > 2 ** 31
    o, lse = ext.forward_varlen(q, k, v, cu, cu, 400, 400, 0.125, causal)
    _same(ext.backward_varlen(do, q, k, v, o, lse, cu, cu, n, n, 0.125, causal),
          ext.backward_varlen(do, q, k, v, o, lse, cu, cu, 400, 400, 0.125, causal))
    assert ext.device_status() == 0
