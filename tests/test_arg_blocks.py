"""The one-block calls of the C ABI: the block layouts of the Python binding and the argument checks behind them."""
import ctypes
import struct

import pytest

ext = pytest.importorskip("flash_attn_legacy_cuda")

INVALID, BAD_HEAD_DIM = -1, -2


def _fwd(heads_q=8, heads_kv=2, d=64, scale=0.125, causal=0, q=256):
    stride = (1 << 16, 1 << 12, 64)
    return ext._FWD_ARGS.pack(q, 256, 256, 256, 256, 0, 1, heads_q, heads_kv, 64, 64, d, *stride * 4, scale, causal, 0, 0)


@pytest.mark.parametrize("bad,code", [({"q": 0}, INVALID), ({"heads_kv": 3}, INVALID), ({"scale": 0.0}, INVALID),
                                      ({"causal": 3}, INVALID), ({"causal": -1}, INVALID), ({"d": 48}, BAD_HEAD_DIM)])
def test_forward_block_goes_through_the_checks_of_fal_fwd(bad, code):
    assert ext._fwd_run(_fwd(**bad)) == code


def test_blocks_of_zeros_and_null_are_refused():
    for run, layout in ((ext._fwd_run, ext._FWD_ARGS), (ext._bwd_run, ext._BWD_ARGS), (ext._decode_run, ext._DECODE_ARGS)):
        assert run(bytes(layout.size)) == INVALID
        assert run(ctypes.c_char_p(None)) == INVALID


@pytest.mark.parametrize("given", ["0.125", 1e39, -1e39, 1e-50, 0.1, 2])
def test_scales_are_converted_as_ctypes_converts_them(given):
    """Whatever float() takes goes into the block as the 32-bit float a C argument would be."""
    want = ctypes.c_float(float(given)).value
    block = _fwd(scale=ext._scale(given))
    assert struct.unpack_from("@f", block, 6 * 8 + 6 * 4 + 12 * 8)[0] == want
    if want <= 0:
        assert ext._fwd_run(block) == INVALID
