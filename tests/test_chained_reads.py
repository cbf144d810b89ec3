"""The cell passes are chained: a kernel's blocks are resident while its
predecessor still writes the counts, prefixes and the list.  What the chain
writes is therefore not read through the read-only path (__ldg), which is for
memory that does not change while the reading kernel runs."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "isosurface_gb300", "csrc")
WRITTEN = ("segs", "masks", "blocks", "list", "ctrl", "totals")


def test_counts_and_lists_are_not_read_as_constants():
    text = open(os.path.join(CSRC, "mc_cells.cuh")).read()
    assert all(re.search(r"A\.(c\.)?%s\b" % name, text) for name in WRITTEN)
    read = re.findall(r"__ldg\(&?A\.(?:c\.)?(\w+)", text)
    assert "seg_grid" in read and not set(read) & set(WRITTEN)
