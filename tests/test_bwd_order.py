"""The order of the backward's GEMMs that the release of its buffers rests on, read from the source."""
import os
import re

from conftest import PKG


def test_dq_is_always_issued_before_the_commit_that_frees_its_operand():
    """At head_dim 256 the commit behind dK hands dS^T's buffer to the next loads; dQ reads it too, so no build
    option may issue dQ behind that commit."""
    with open(os.path.join(PKG, "csrc", "fal_bwd.cu")) as f:
        source = f.read()
    calls = [(m.start(), m.group(1)) for m in re.finditer(r"^\s*issue_(dq|dk)\(\);", source, re.M)]
    assert [name for _, name in calls] == ["dq", "dk"]
    body = source[source.rindex("auto issue_dk", 0, calls[0][0]):source.index("\n", calls[1][0])]
    assert "tc_commit(bar(iQEmpty + st))" in body
    assert not re.search(r"^\s*#\s*(if|else|elif)", body, re.M)
