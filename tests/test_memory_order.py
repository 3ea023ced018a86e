"""Source checks on what orders memory accesses between dependent launches
(csrc/pdl.cuh): a kernel that may come up while the one before it still runs
reads nothing before its griddepcontrol.wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "sse_wilson_dslash_gb300", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_assembly_that_reads_global_memory_is_ordered(path):
    """An asm statement that is neither volatile nor clobbers memory is a pure
    function of its operands to the compiler, which may move it above the wait."""
    text = open(path).read()
    for m in re.finditer(r"\basm\b(\s+volatile)?\s*\(((?:[^;]|;(?!\n))*?)\);", text):
        if re.search(r"\bld\.(global|const|relaxed|acquire|weak|volatile)|\bcp\.async|\bprefetch", m.group(2)):
            assert m.group(1) or '"memory"' in m.group(2), m.group(0)
