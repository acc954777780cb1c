"""The forward's choice of a CTA shape, compiled from its source for 148 SMs, against the shape that measured faster."""
import ctypes
import os
import re
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

AUTO, ONE, TWO, HALF = 0, 1, 2, 3
NONE, CAUSAL, END = 0, 1, 2


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    compiler = os.environ.get("CXX", "g++")
    if shutil.which(compiler) is None:
        pytest.skip("no C++ compiler")
    with open(os.path.join(PKG, "csrc", "fal_api.cu")) as f:
        source = f.read()
    rules = source[source.index("std::atomic<int> g_fwd_variant"):source.index("// CTAs that share the keys of each")]
    (call,) = re.findall(r"^  int variant = (forward_variant\(.*?\));", source, re.S | re.M)
    (packed,) = re.findall(r"const int variant = (forward_variant\(.*?\));", source, re.S | re.M)
    folder = tmp_path_factory.mktemp("shape")
    text = f"""#include <atomic>
#include <cstdint>
#include "fal_b200.h"
static int sm_count() {{ return 148; }}
{rules}
extern "C" int batched(int kdim, int seqlen_q, int seqlen_k, int batch, int heads_q, int is_causal) {{ return {call}; }}
extern "C" int packed(int kdim, int total_q, int total_k, int num_seqs, int heads_q, int is_causal) {{ return {packed}; }}
"""
    (folder / "shape.cpp").write_text(text)
    subprocess.run([compiler, "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "include"),
                    str(folder / "shape.cpp"), "-o", str(folder / "shape.so")], check=True)
    return ctypes.CDLL(str(folder / "shape.so"))


# units x rows of head_dim 64: whichever shape was faster by more than two runs differ (times at half_sm_pays)
@pytest.mark.parametrize("units,rows,mask,best", [
    (16, 4000, CAUSAL, TWO), (16, 4096, CAUSAL, TWO), (17, 4000, CAUSAL, TWO), (20, 3000, CAUSAL, TWO), (24, 3000, CAUSAL, TWO),
    (24, 2500, CAUSAL, TWO), (32, 2048, CAUSAL, TWO), (36, 1700, CAUSAL, TWO), (24, 2900, CAUSAL, TWO),
    (8, 4000, CAUSAL, ONE), (16, 2100, CAUSAL, ONE), (17, 2100, CAUSAL, ONE), (14, 2650, CAUSAL, ONE),
    (12, 4000, CAUSAL, HALF), (16, 3000, CAUSAL, HALF), (18, 3072, CAUSAL, HALF), (27, 2100, CAUSAL, HALF), (40, 1600, CAUSAL, HALF),
    (48, 2600, CAUSAL, HALF), (48, 4000, CAUSAL, HALF), (33, 2304, CAUSAL, HALF), (81, 257, CAUSAL, HALF), (54, 577, CAUSAL, HALF),
    (32, 1143, CAUSAL, HALF), (100, 400, CAUSAL, HALF),
    (32, 2048, NONE, TWO), (36, 2048, NONE, TWO), (54, 2048, NONE, TWO), (88, 2048, NONE, TWO), (48, 1500, NONE, TWO),
    (64, 1000, NONE, TWO), (72, 700, NONE, HALF), (96, 700, NONE, TWO), (72, 1300, NONE, TWO),
    (25, 2048, NONE, HALF), (64, 2048, NONE, HALF), (50, 1024, NONE, HALF), (252, 1024, NONE, HALF), (109, 577, NONE, HALF),
    (130, 257, NONE, HALF), (289, 200, NONE, HALF), (16, 2048, NONE, TWO), (32, 1600, NONE, HALF),
])
def test_rows_of_one_length(choose, units, rows, mask, best):
    assert choose.batched(64, rows, rows, units, 1, mask) == best


@pytest.mark.parametrize("lengths,heads,mask,best", [
    ([992] * 24, 16, NONE, HALF), ([1694] * 12, 16, NONE, HALF), ([1267] * 42, 16, NONE, HALF), ([1485] * 7, 16, NONE, TWO),
    ([1743] * 9, 8, NONE, TWO), ([1174] * 6, 8, NONE, TWO), ([1527] * 4, 16, NONE, TWO), ([1083] * 2, 16, CAUSAL, ONE),
    ([302] * 5, 16, CAUSAL, HALF), ([2048] * 8, 16, NONE, TWO), ([3500] * 6, 16, NONE, TWO),
    ([992] * 24, 16, CAUSAL, HALF), ([2048] * 8, 16, CAUSAL, HALF), ([81] * 10, 16, CAUSAL, HALF),
])
def test_packed(choose, lengths, heads, mask, best):
    total = sum(lengths)
    assert choose.packed(64, total, total, len(lengths), heads, mask) == best


def test_every_head_dim_has_a_shape(choose):
    for kdim in (64, 128, 256):
        for units in (1, 7, 40, 150, 1000):
            for rows in (1, 128, 129, 700, 5000):
                for mask in (NONE, CAUSAL, END):
                    shape = choose.batched(kdim, rows, rows, units, 1, mask)
                    assert shape == ONE if kdim == 256 else shape in ((ONE, TWO, HALF) if kdim == 64 else (ONE, TWO))
