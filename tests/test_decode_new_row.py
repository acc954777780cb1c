"""Decode with a new token: which slices of an entry load with the choice of a row's source, read from the source."""
import os
import re

import pytest

from conftest import PKG


@pytest.mark.parametrize("new_local", [-1, 0, 1, 15, 16, 17, 1999, 2047, 2048, 7999])
def test_only_the_slice_with_the_new_row_chooses_its_source(new_local):
    """The choice costs every load of the slice that makes it, so the slices without the row must not."""
    with open(os.path.join(PKG, "csrc", "fal_decode.cu")) as f:
        source = f.read()
    keys = int(re.search(r"constexpr int kSliceKeys = (\d+);", source).group(1))
    ((condition, variant),) = re.findall(r"^\s*if \((.+)\) load\(std::(true|false)_type\{\}\);", source, re.M)
    condition = re.sub(r"static_cast<unsigned>\((.+?)\)", r"((\1) % 2**32)", condition)
    chosen = [key0 for key0 in range(0, max(new_local + 1, 1), keys)
              if eval(condition, {"new_local": new_local, "key0": key0, "kSliceKeys": keys}) == (variant == "true")]
    assert chosen == ([new_local // keys * keys] if new_local >= 0 else [])
