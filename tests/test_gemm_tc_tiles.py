"""A tensor-core product's extents and its kernel come from one table: a kernel launched
with another tile's boxes and stage bytes would write out of range, which no test may
provoke.  So the source is what is checked: kernels are instantiated in the table's
entries and nowhere else, from the extents the entry states."""
import os
import re

from conftest import PACKAGE


def test_kernels_are_named_in_the_table_only():
    with open(os.path.join(PACKAGE, "csrc", "gemm_tc.cu")) as source:
        text = source.read()
    begin = text.index("constexpr TcTile make_tile()")
    end = text.index("\n}\n", begin)
    named = [m.start() for m in re.finditer(r"gemm_tc_kernel\s*<", text)]
    assert named and all(begin < at < end for at in named)
    for m in re.finditer(r"gemm_tc_kernel\s*<([^>]*)>", text):
        assert m.group(1).split(",")[:2] == ["M", " N"]
    assert "TcTile tile = {M, N," in text[begin:end]
