"""Rules that the kernels' sources keep, read as text (no GPU)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmt_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_read_only_loads_in_programmatic_dependents(path):
    """A kernel launched as a programmatic dependent is resident while the one before it still writes its inputs, so memory
    must not be read through the read-only path: neither by name nor by parameters from which the compiler infers it."""
    code = re.sub(r"//[^\n]*", "", open(path).read())
    assert "__ldg(" not in code
    assert not re.search(r"\bld\.global(\.\w+)*\.nc\b", code)
    assert not re.search(r"\bconst\s+[\w:]+\s*\*\s*__restrict__", code)
